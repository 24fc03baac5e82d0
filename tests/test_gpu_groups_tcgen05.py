"""Group sums on tcgen05 (widths that are no multiple of 512, and blocks off the 16-byte grid) at the edges of its tiles."""

import numpy as np
import pytest
import torch

from oracle import tq1_oracle as o
from tests.gpu_util import random_blocks, run_linear, to_dev

pytestmark = pytest.mark.gpu

# Relative error (2-norm): two truncating steps per accumulator, on average half an ulp of 0.72 * 2^-23 each of a value that
# grows from zero (0.96 * 2^-24), two FP32 additions of four accumulators (0.58 * 2^-24 each, in quadrature 0.82), and one
# rounding of the carried sum (0.58).
BOUND = (0.96 + 0.82 + 0.58) * 2.0 ** -24


@pytest.mark.parametrize(("rows", "columns", "batch"), (
    (9000, 3200, 12), (17408, 3200, 16),                # one unit, of 16 tokens; a cluster of 2
    (17408, 1664, 17), (14000, 2688, 32),               # of 32, rows that fill no tile
    (17408, 1408, 24), (38000, 1408, 24),               # one unit and an odd number of groups, in one tile and in three
    (4099, 2176, 33), (1500, 5248, 48), (383, 4224, 255),       # two units, clusters of 4, 8 and 8
    (4099, 2176, 65), (9000, 640, 129), (13313, 384, 200)))        # several token tiles, more tiles than SMs, three groups
@pytest.mark.parametrize("shift", (0, 4))
def test_against_float64(rows, columns, batch, shift):
    from ternel_b200.dispatch import plan
    from ternel_b200.ops import check_status, tq1_get_rows, tq1_matmul
    assert plan(batch, rows, columns).form == "groups_tcgen05"
    blocks, rng = random_blocks(rows, columns, seed=rows + batch)
    backing = torch.zeros(blocks.size + 16, dtype=torch.uint8, device="cuda")
    bd = backing[shift:shift + blocks.size].view(blocks.shape)
    bd.copy_(torch.from_numpy(blocks))
    x = torch.from_numpy(rng.standard_normal((batch, columns)).astype(np.float16)).cuda()
    dense = tq1_get_rows(bd, torch.arange(rows, device="cuda"), dtype=torch.float32).double()
    want = x.double() @ dense.T
    got = tq1_matmul(bd, x, out_dtype=torch.float32)
    assert float((got.double() - want).norm() / want.norm()) <= BOUND
    assert torch.equal(tq1_matmul(bd, x, out_dtype=torch.float32), got)
    assert torch.equal(tq1_matmul(bd, x), got.half())
    check_status()


@pytest.mark.parametrize(("rows", "columns", "batch", "form"), (
    (17408, 3200, 12, "tcgen05"), (17408, 1408, 32, "tcgen05"),         # one unit, CTAs by themselves
    (4099, 2176, 48, "tcgen05"), (4099, 2176, 129, "tcgen05"),          # a cluster of 4, several token tiles
    (16500, 640, 16, "many"), (9000, 640, 100, "many")))
@pytest.mark.parametrize("kind", ("scales", "activations", "infinite sum"))
def test_nonfinite_values(rows, columns, batch, form, kind):
    """Whole activations: infinities of a sum's sign, NaN for 0 * Inf and Inf - Inf, and a sum that has become infinite stays so."""
    from ternel_b200.dispatch import plan
    assert plan(batch, rows, columns).form == "groups_" + form
    blocks, rng = random_blocks(rows, columns, seed=batch)
    x = rng.integers(-3, 4, (batch, columns)).astype(np.float16)
    scales = blocks.reshape(rows, columns // 128, 28)[:, :, :2].copy().view(np.float16)[:, :, 0]
    if kind == "scales":
        hit = rng.random(scales.shape) < 0.1
        scales[hit] = rng.choice(np.array([np.inf, -np.inf, np.nan, 0.0], dtype=np.float16), hit.sum())
    elif kind == "activations":
        hit = rng.random(x.shape) < 0.5 / columns
        x[hit] = rng.choice(np.array([np.inf, -np.inf, np.nan], dtype=np.float16), hit.sum())
    else:
        scales[:, 0], x[0, :128] = np.inf, 1.0
    blocks[:, :, :2] = scales[:, :, None].copy().view(np.uint8)
    few = rng.choice(rows, 300, replace=False)          # the oracle takes its time
    with np.errstate(invalid="ignore", over="ignore"):
        want = o.reference_matmul(np.ascontiguousarray(blocks[few]), x.astype(np.float32), rows=300, columns=columns)
    got = run_linear(blocks, x)[:, few]
    assert not np.isfinite(want).all()
    assert np.array_equal(o.nonfinite_classes(got), o.nonfinite_classes(want))


def test_without_a_workspace_nothing_waits():
    """A caller without a status word cannot be told that a wait ran out, so its calls stay on the forms that have none: the
    results are those of a few tokens at a time, which take the same sums in the same order."""
    from ternel_b200 import _native
    rows, columns, batch = 4099, 2176, 64
    blocks, rng = random_blocks(rows, columns, seed=5)
    x = rng.standard_normal((batch, columns)).astype(np.float16)
    bd, xd = to_dev(blocks), to_dev(x)
    y = torch.empty((batch, rows), dtype=torch.float32, device="cuda")
    assert _native.lib().tq1_linear_f16(bd.data_ptr(), xd.data_ptr(), y.data_ptr(), 1, batch, rows, columns, None, 0,
                                        torch.cuda.current_stream().cuda_stream) == 0
    got = y.cpu().numpy()
    assert np.array_equal(got, np.concatenate([run_linear(blocks, x[i:i + 8]) for i in range(0, batch, 8)]))
    with_workspace = run_linear(blocks, x)
    assert not np.array_equal(got, with_workspace)
    assert np.linalg.norm(got - with_workspace) <= 2 * 2.3e-7 * np.linalg.norm(got)       # the forms' bounds


@pytest.mark.parametrize(("rows", "columns", "batch"), ((8192, 8320, 12), (8192, 8320, 24), (8192, 8320, 32), (5120, 17280, 24)))
def test_long_calls_of_nine_to_32_tokens_take_it(rows, columns, batch):
    """Where this form is faster by a quarter it has to be the one that runs: the sums are not those of the form for a caller
    without a workspace, and no less exact."""
    from ternel_b200 import _native
    from ternel_b200.ops import tq1_get_rows, tq1_matmul
    from ternel_b200.stack import random_blocks_device
    gen = torch.Generator(device="cuda")
    gen.manual_seed(6)
    bd = random_blocks_device(rows, columns, gen, "cuda")
    x = torch.randn((batch, columns), generator=gen, device="cuda").half()
    other = torch.empty((batch, rows), dtype=torch.float32, device="cuda")
    assert _native.lib().tq1_linear_f16(bd.data_ptr(), x.data_ptr(), other.data_ptr(), 1, batch, rows, columns, None, 0,
                                        torch.cuda.current_stream().cuda_stream) == 0
    got = tq1_matmul(bd, x, out_dtype=torch.float32)
    assert not torch.equal(got, other)
    want = x.double() @ tq1_get_rows(bd, torch.arange(rows, device="cuda"), dtype=torch.float32).double().T
    assert float((got.double() - want).norm() / want.norm()) <= BOUND
