"""Kernels that are launched while the one before them ends read what it wrote, and write nothing that it still reads."""

import numpy as np
import pytest
import torch

from tests.gpu_util import random_blocks, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("batch", "columns"), (
    (1, 640),           # row kernel
    (5, 640),           # group sums, few rows
    (70, 1408),         # group sums, many rows
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
