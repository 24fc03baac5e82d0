"""Which kernel and tiling a linear call takes, and the recorded sweep the rule was chosen from.

The reference chooses its kernel configuration per batch size from committed sweeps and replays
them in its tests (``select_lut23`` / ``select_gemm``, src/ternel_mlx/modules.py:331-422;
tests/test_mlx_modules.py:553-1084). Here the choice lives in the C library (``tq1_linear_plan``)
and the sweep it was chosen from is ``dispatch_sweep_b200.json`` beside this file:

    python -m ternel_b200.dispatch --out ternel_b200/dispatch_sweep_b200.json    # on a B200

records, for every batch size and shape of the sweep, the time of every token tile the
tensor-core kernel can run with, for batches up to ``LOOPED_MAX`` the time of the same call
as passes of the batch-1 kernel in one launch, for batches of 3 to 16 that of the slice kernel,
and for shapes that are no multiple of 512 wide that of every form of the group sums;
``tests/test_dispatch_replay.py`` checks that the rule's choice is within a few percent of the
best recorded one everywhere.
"""

from __future__ import annotations

import argparse
import ctypes
import json
from dataclasses import dataclass
from pathlib import Path

from . import _native
from .format import check

SWEEP_PATH = Path(__file__).resolve().parent / "dispatch_sweep_b200.json"
KERNELS = {0: "rows", 1: "stream_gemv", 2: "tensor_core", 3: "group_sums"}
FORMS = {0: "rows", 1: "stream_gemv", 2: "tcgen05", 3: "slices", 4: "groups_few", 5: "groups_many", 6: "groups_tcgen05"}
TOKEN_TILES = (16, 32, 64, 128, 256)
LOOPED_MAX = 4          # largest batch also timed as passes of the batch-1 kernel
SWEEP_BATCHES = (2, 3, 4, 8, 16, 17, 24, 32, 33, 48, 64, 65, 96, 128, 192, 256, 512, 1023, 1024, 2048)
SWEEP_SHAPES = ((5120, 5120), (1024, 5120), (17408, 5120), (5120, 17408))
GROUP_BATCHES = (9, 12, 16, 17, 24, 32, 33, 48, 64, 100, 129, 300)
GROUP_SHAPES = ((383, 4224), (4099, 2176), (5120, 640), (5120, 5248), (8192, 8320), (5120, 17280), (13313, 640), (17408, 5248))


@dataclass(frozen=True)
class LinearPlan:
    kernel: str          # "rows", "stream_gemv", "tensor_core" or "group_sums"
    token_tile: int      # activation rows per tile (tensor-core kernel), else 0
    ctas: int
    parts: int           # equal K parts per tile, 0 = stream-K ranges
    form: str            # the kernel that runs, one of FORMS: "slices" takes some of "tensor_core"'s calls of up to 16 rows
                         # (the tile, CTAs and parts are the tcgen05 kernel's), and "group_sums" has three. ring_layout() tells the
                         # two kernels of "stream_gemv" apart, and how the tcgen05 kernel's parts are added up


def plan(batch: int, rows: int, columns: int, *, aligned: bool = True, workspace: bool = True) -> LinearPlan:
    """The library's choice for ``x[batch, columns] @ W[rows, columns].T`` (launches nothing)."""
    kernel, tile, ctas, parts, form = (ctypes.c_int() for _ in range(5))
    lib = _native.lib()
    check(lib.tq1_linear_plan(batch, rows, columns, int(aligned), ctypes.byref(kernel), ctypes.byref(tile),
                              ctypes.byref(ctas), ctypes.byref(parts)))
    check(lib.tq1_linear_form(batch, rows, columns, int(aligned), int(workspace), ctypes.byref(form)))
    return LinearPlan(KERNELS[kernel.value], tile.value, ctas.value, parts.value, FORMS[form.value])


@dataclass(frozen=True)
class RingLayout:
    cluster: int         # CTAs that share a row tile's columns
    sets: int            # sets of warps that take turns on the row tiles
    stages: int          # row tiles that a CTA holds at a time
    tiles: int           # row tiles of a cluster
    preferred: bool      # what the rules say: of one row, this kernel or a chain of one link; of three to sixteen, this one or tcgen05


def ring_layout(form: str, batch: int, rows: int, columns: int, *, rooms: "dict[int, int] | None" = None) -> "RingLayout | None":
    """How the kernel that streams row tiles for 1 and 2 activation rows (``"stream_gemv"``) or that for 3 to 16 (``"slices"``) lays out
    a call, whether or not the rules send it there; None where it does not take it (a batch-1 call then is a chain of one link).
    ``"tcgen05"``: the parts of an output tile as ``sets``, and in ``cluster`` the CTAs that add them up, 1 where they meet in the
    workspace. ``rooms`` replaces what the driver says of how many clusters of a size run at once."""
    ask = _native.lib().tq1_debug_call_layout
    ask.restype, ask.argtypes = ctypes.c_int, [ctypes.c_int] * 4 + [ctypes.c_void_p] * 2
    given = (ctypes.c_int * 17)(*(rooms.get(size, 0) for size in range(17))) if rooms is not None else None
    out = (ctypes.c_int * 5)()
    check(ask({name: number for number, name in FORMS.items()}[form], batch, rows, columns, given, out))
    return RingLayout(*out[:4], bool(out[4])) if out[0] else None


def looped_tokens() -> int:
    """Largest batch the library runs as passes of the batch-1 kernel (found by probing the plan)."""
    tokens = 1
    while tokens < 8 and plan(tokens + 1, 5120, 5120).kernel == "stream_gemv":
        tokens += 1
    return tokens


def chosen_over_best(case: dict) -> "tuple[float, LinearPlan]":
    """Recorded time of the library's choice for a sweep case over the best recorded option of that case."""
    tiles = {int(k): v for k, v in case.get("us_by_token_tile", {}).items()}
    forms = case.get("us_by_form", {})
    best = min([*tiles.values(), *forms.values(), *([case["us_looped"]] if "us_looped" in case else [])])
    chosen = plan(case["batch"], case["rows"], case["columns"])
    took = (case["us_looped"] if chosen.form == "stream_gemv" else
            tiles[chosen.token_tile] if chosen.form == "tcgen05" else forms[chosen.form])
    return took / best, chosen


def load_sweep(path: Path = SWEEP_PATH) -> dict:
    return json.loads(Path(path).read_text())


def record_sweep(batches=SWEEP_BATCHES, shapes=SWEEP_SHAPES, tiles=TOKEN_TILES, group_batches=GROUP_BATCHES,
                 group_shapes=GROUP_SHAPES, replays: int = 3) -> dict:
    """Time every (batch, shape, token tile or form) on the current GPU: CUDA-graph replays over a ring of distinct weight
    buffers of more than twice the L2 cache, so that every call reads its weights from HBM, CUDA events. Returns the
    JSON-ready record."""
    import torch
    from .stack import random_blocks_device

    default_loop = looped_tokens()
    lib = _native.lib()
    lib.tq1_debug_set_loop_tokens.restype = ctypes.c_int
    lib.tq1_debug_set_loop_tokens.argtypes = [ctypes.c_int]
    lib.tq1_debug_linear_as.restype = ctypes.c_int
    lib.tq1_debug_linear_as.argtypes = [ctypes.c_int, *_native.SIGNATURES["tq1_linear_f16"][1][:8], ctypes.c_void_p]
    form_number = {name: number for number, name in FORMS.items()}
    device = torch.device("cuda")
    gen = torch.Generator(device=device)
    gen.manual_seed(7)
    cases, group_cases = [], []

    def ring_of(rows, columns):
        packed = random_blocks_device(rows, columns, gen, device)
        ring = 2 * torch.cuda.get_device_properties(device).L2_cache_size // packed.numel() + 1
        return [packed.clone() for _ in range(ring)]

    def vectors(batch, rows, columns):
        return (torch.randn((batch, columns), generator=gen, device=device).to(torch.float16),
                torch.empty((batch, rows), dtype=torch.float16, device=device))

    def time_call(weights, x, y, batch, rows, columns, form=None):
        need = lib.tq1_linear_workspace_bytes(batch, rows, columns)
        ws = torch.zeros(need, dtype=torch.uint8, device=device)

        def run():
            stream = ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)
            for w in weights:
                if form is None:
                    check(lib.tq1_linear_f16(w.data_ptr(), x.data_ptr(), y.data_ptr(), 0, batch, rows, columns,
                                             ws.data_ptr(), need, stream))
                else:
                    check(lib.tq1_debug_linear_as(form_number[form], w.data_ptr(), x.data_ptr(), y.data_ptr(), 0, batch, rows,
                                                  columns, ws.data_ptr(), stream))

        torch.cuda.synchronize()
        side = torch.cuda.Stream(device=device)
        with torch.cuda.stream(side):
            run()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        graph.replay()
        start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        start.record()
        for _ in range(replays):
            graph.replay()
        stop.record()
        torch.cuda.synchronize()
        del graph
        return round(start.elapsed_time(stop) * 1e3 / (replays * len(weights)), 3)

    try:
        for rows, columns in shapes:
            weights = ring_of(rows, columns)
            for batch in batches:
                x, y = vectors(batch, rows, columns)
                times = {}
                check(lib.tq1_debug_set_loop_tokens(0))        # the tensor-core kernel, tile by tile
                for tile in tiles:
                    if tile > 16 and tile >= 4 * batch:       # a tile mostly of padding: not a candidate
                        continue
                    check(lib.tq1_debug_force_token_tile(tile))
                    times[str(tile)] = time_call(weights, x, y, batch, rows, columns)
                case = {"batch": batch, "rows": rows, "columns": columns, "us_by_token_tile": times}
                if batch <= LOOPED_MAX:                        # the same call as passes of the batch-1 kernel
                    check(lib.tq1_debug_force_token_tile(0))
                    check(lib.tq1_debug_set_loop_tokens(batch))
                    case["us_looped"] = time_call(weights, x, y, batch, rows, columns)
                if 3 <= batch <= 16:
                    case["us_by_form"] = {"slices": time_call(weights, x, y, batch, rows, columns, "slices")}
                cases.append(case)
            del weights
        for rows, columns in group_shapes:
            weights = ring_of(rows, columns)
            for batch in group_batches:
                x, y = vectors(batch, rows, columns)
                group_cases.append({"batch": batch, "rows": rows, "columns": columns, "us_by_form": {
                    form: time_call(weights, x, y, batch, rows, columns, form)
                    for form in ("groups_few", "groups_many", "groups_tcgen05")}})
            del weights
    finally:
        check(lib.tq1_debug_force_token_tile(0))
        check(lib.tq1_debug_set_loop_tokens(default_loop))
    return {"device": torch.cuda.get_device_name(device), "unit": "microseconds per call, CUDA-graph replays, distinct weight buffers of more than twice L2", "cases": cases,
            "group_cases": group_cases}


def main() -> None:
    parser = argparse.ArgumentParser(description=__doc__.split("\n\n")[0])
    parser.add_argument("--out", type=Path, default=SWEEP_PATH)
    args = parser.parse_args()
    record = record_sweep()
    args.out.write_text(json.dumps(record, indent=1) + "\n")
    every = record["cases"] + record["group_cases"]
    worst = max(chosen_over_best(case)[0] for case in every)
    print(f"wrote {args.out} ({len(every)} cases); the rule's worst case is {worst:.3f}x the best recorded option")


if __name__ == "__main__":
    main()
