"""The batched kernels for widths that are no multiple of 512 and for blocks off the 16-byte grid: an FP32 sum per group,
scaled once, as the reference does it. Needs a B200."""

import numpy as np
import pytest
import torch

from oracle import tq1_oracle as o
from tests.gpu_util import random_blocks, run_linear, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", (2, 8, 9, 16, 17, 32, 33, 64, 65, 129))
@pytest.mark.parametrize(("rows", "columns"), ((4099, 2176), (383, 4224), (8191, 128), (13313, 640), (16500, 1408), (1000, 5248)))
def test_error_of_group_sums(rows, columns, batch):
    """Every token tile of both kernels, on both sides of the lines between them, rows and groups that fill no tile. With n
    roundings in a row the result's relative error (2-norm) is about sqrt(n / 3) * 2^-24; n is at most 4 in a group and 41
    over the groups, so 2.3e-7. (One truncating accumulator over the columns was at 1.3e-6 for 2176 of them.)"""
    if batch * rows * columns < 1 << 20:
        pytest.skip("the row kernel's")
    from ternel_b200.dispatch import plan
    from ternel_b200.ops import tq1_get_rows, tq1_matmul
    assert plan(batch, rows, columns).kernel == "group_sums"
    blocks, rng = random_blocks(rows, columns, seed=rows + batch, dist="tests")
    bd, x = to_dev(blocks), torch.from_numpy(rng.standard_normal((batch, columns)).astype(np.float16)).cuda()
    dense = tq1_get_rows(bd, torch.arange(rows, device="cuda"), dtype=torch.float32).double()
    want = x.double() @ dense.T
    got = tq1_matmul(bd, x, out_dtype=torch.float32)
    assert float((got.double() - want).norm() / want.norm()) < 2.3e-7
    assert torch.equal(tq1_matmul(bd, x, out_dtype=torch.float32), got)
    assert torch.equal(tq1_matmul(bd, x), got.half())


def test_blocks_off_the_16_byte_grid():
    rows, columns, batch = 1500, 1024, 20
    blocks, rng = random_blocks(rows, columns, seed=3, dist="tests")
    x = rng.standard_normal((batch, columns)).astype(np.float16)
    from ternel_b200.ops import tq1_matmul
    for shift in (4, 8, 12):
        backing = torch.zeros(blocks.size + 16, dtype=torch.uint8, device="cuda")
        shifted = backing[shift:shift + blocks.size].view(blocks.shape)
        shifted.copy_(torch.from_numpy(blocks))
        got = tq1_matmul(shifted, to_dev(x), out_dtype=torch.float32).cpu().numpy()
        want = o.float64_matmul(blocks, x.astype(np.float32), rows=rows, columns=columns)
        assert np.linalg.norm(got - want) < 2.3e-7 * np.linalg.norm(want)


@pytest.mark.parametrize(("rows", "columns", "batch"), ((300, 640, 7), (300, 640, 16), (200, 1408, 31), (4800, 640, 70), (16400, 128, 12)))
@pytest.mark.parametrize("kind", ("scales", "activations", "infinite sum"))
def test_nonfinite_values_come_out_as_in_the_reference_order(rows, columns, batch, kind):
    """Whole activations, so that every group sum is exact in any order: an infinite scale times a group's sum is an
    infinity of the sum's sign, NaN where the sum is zero; 0 * Inf and Inf - Inf are NaN; a sum that has become
    infinite stays so in the groups after it."""
    assert batch * rows * columns >= 1 << 20
    blocks, rng = random_blocks(rows, columns, seed=rows + batch, dist="tests")
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
    with np.errstate(invalid="ignore", over="ignore"):
        want = o.reference_matmul(blocks, x.astype(np.float32), rows=rows, columns=columns)
    got = run_linear(blocks, x)
    assert not np.isfinite(want).all()
    assert np.array_equal(o.nonfinite_classes(got), o.nonfinite_classes(want))
