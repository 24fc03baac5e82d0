"""The library's kernel/tile choice replayed against the recorded B200 sweep (no GPU needed): for every
recorded (batch, shape) the chosen token tile must be within 10% of the best recorded one, the way the
reference replays its dispatch rules against committed sweeps (tests/test_mlx_modules.py:553-1084 there)."""

import pytest

from ternel_b200.dispatch import (GROUP_BATCHES, GROUP_SHAPES, LOOPED_MAX, SWEEP_BATCHES, SWEEP_SHAPES, chosen_over_best,
                                  load_sweep, plan)


def test_rule_is_near_the_best_recorded_option_everywhere():
    sweep = load_sweep()
    assert len(sweep["cases"]) == len(SWEEP_BATCHES) * len(SWEEP_SHAPES)
    worst = 1.0
    for case in sweep["cases"]:
        assert ("us_looped" in case) == (case["batch"] <= LOOPED_MAX)       # every arm recorded where it exists
        assert ("us_by_form" in case) == (3 <= case["batch"] <= 16)
        ratio, chosen = chosen_over_best(case)
        assert chosen.kernel in ("tensor_core", "stream_gemv")
        assert ratio <= 1.10, (case, chosen)
        worst = max(worst, ratio)
    assert 1.0 <= worst <= 1.10


def test_plan_boundaries():
    assert plan(1, 5120, 5120).kernel == "stream_gemv"
    assert plan(1, 5120, 5120, aligned=False).kernel == "rows"
    assert plan(1, 5120, 640).kernel == "rows"                 # K not a multiple of 512
    assert plan(4, 100, 640).kernel == "rows"
    assert plan(2, 17408, 5120).kernel == "stream_gemv"       # two passes of the batch-1 kernel in one launch
    small = plan(5, 17408, 5120)
    assert (small.kernel, small.token_tile, small.parts) == ("tensor_core", 16, 2) and small.ctas == 272
    for batch in range(5, 17):
        assert plan(batch, 5120, 17408).token_tile == 16       # up to 16 rows: always the 16-row tile
    big = plan(2048, 17408, 5120)
    assert big.token_tile == 256 and big.parts == 0 and big.ctas == 148       # stream-K over one CTA per SM
    assert plan(192, 17408, 5120).token_tile == 256            # one 256-row tile beats two 128-row tiles
    with pytest.raises(ValueError):
        plan(0, 128, 512)


def test_two_rows_of_any_matrix_take_the_exact_kernel():
    """Two activation rows of every matrix that the batch-1 kernel takes are two passes of it (exact integer group
    sums), and recording a sweep leaves that rule as it found it."""
    import ctypes
    from ternel_b200 import _native
    from ternel_b200.dispatch import looped_tokens
    shapes = [(16, 512), (1024, 5120), (5120, 5120), (4096, 4096), (17408, 5120)]
    assert looped_tokens() == 2
    for rows, columns in shapes:
        assert plan(2, rows, columns).kernel == "stream_gemv"
        assert plan(3, rows, columns).kernel == "tensor_core"
    setter = _native.lib().tq1_debug_set_loop_tokens           # what record_sweep does around its timings
    setter.argtypes, before = [ctypes.c_int], looped_tokens()
    assert setter(0) == 0 and plan(2, 17408, 5120).kernel == "tensor_core"
    assert setter(before) == 0
    for rows, columns in shapes:
        assert plan(2, rows, columns).kernel == "stream_gemv"


def test_two_rows_that_neither_exact_kernel_takes_are_planned_as_they_run():
    """More rows than two links have slots for: the tile kernel, where it has room for the columns; else the batched one."""
    assert plan(2, 151936, 5120).kernel == "stream_gemv"
    assert plan(2, 9008, 65536).kernel == plan(2, 9008, 65536).form.replace("tcgen05", "tensor_core") == "tensor_core"
    assert plan(2, 8192, 65536).kernel == plan(1, 9008, 65536).kernel == "stream_gemv"


def test_rule_between_the_forms_of_the_group_sums():
    """The line is drawn by times behind another kernel, where the tcgen05 form begins 1 to 2 us later than it does in the recorded
    rows of calls: up to 20% of the shortest calls (383 rows), 10% of the others."""
    cases = load_sweep()["group_cases"]
    assert len(cases) == len(GROUP_BATCHES) * len(GROUP_SHAPES)
    for case in cases:
        ratio, chosen = chosen_over_best(case)
        assert chosen.kernel == "group_sums"
        assert ratio <= (1.20 if case["rows"] < 1000 else 1.10), (case, chosen)


def test_plan_names_the_kernel_that_runs():
    assert plan(1, 5120, 5120).form == plan(2, 5120, 5120).form == "stream_gemv"
    assert plan(1, 5120, 640).form == plan(4, 100, 640).form == "rows"
    for batch in range(3, 9):                                  # few rows: mma.sync out of registers, not tcgen05
        assert plan(batch, 1024, 5120).form == "slices" and plan(batch, 1024, 5120).kernel == "tensor_core"
    assert plan(8, 34816, 512).form == plan(16, 17408, 5120).form == plan(17, 1024, 5120).form == "tcgen05"
    assert plan(8, 4099, 2176).form == plan(16, 4099, 2176).form == "groups_few"
    assert plan(16, 34816, 640).form == "groups_many"
    for batch in (12, 32, 300):                                # without a status word nothing may wait
        assert plan(batch, 8192, 8320).form == "groups_tcgen05"
        assert plan(batch, 8192, 8320, workspace=False).form in ("groups_few", "groups_many")
    assert plan(8, 1024, 5120, aligned=False).form == "groups_few"
