"""The host codec when there is no memory for its threads (host code only)."""

import subprocess
from pathlib import Path

from ternel_b200.build import LIB_PATH

PROGRAM = r"""
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <atomic>
#include <new>
#include <vector>
#include "ternel_b200.h"

static std::atomic<bool> empty{false};
void *operator new(std::size_t n) {                 // the library's allocations come here too
    if (empty.load()) throw std::bad_alloc();
    if (void *p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, std::size_t) noexcept { free(p); }

int main() {
    const int64_t groups = 40961, tile = 1;
    std::vector<uint8_t> scales(groups * 2, 7), trits(groups * 128), blocks(groups * 28), back(groups * 128), s2(groups * 2);
    std::vector<uint8_t> codes(groups * 26), again(groups * 28);
    std::vector<uint16_t> halves(groups);
    for (size_t i = 0; i < trits.size(); ++i) trits[i] = (uint8_t)((i * 2654435761u >> 13) % 3);
    int64_t a = 0, b = 0;
    empty = true;
    if (tq1_pack_blocks(scales.data(), trits.data(), blocks.data(), groups, &a) != TQ1_OK) return 2;
    if (tq1_unpack_blocks(blocks.data(), s2.data(), back.data(), groups, 1, &a, &b) != TQ1_OK) return 3;
    if (tq1_tile_blocks(blocks.data(), codes.data(), halves.data(), groups, 1, tile) != TQ1_OK) return 4;
    if (tq1_untile_blocks(codes.data(), halves.data(), again.data(), groups, 1, tile) != TQ1_OK) return 5;
    empty = false;
    if (back != trits || s2 != scales || again != blocks) return 6;
    puts("fine");
    return 0;
}
"""


def test_work_is_done_without_threads_when_there_is_no_memory_for_them(tmp_path):
    """Whatever keeps a thread from starting, its part is done by the caller: nothing is thrown through the C ABI."""
    include = Path(__file__).resolve().parents[1] / "include"
    source, program = tmp_path / "memory.cpp", tmp_path / "memory"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{include}", str(source), "-o", str(program), str(LIB_PATH),
                    f"-Wl,-rpath,{LIB_PATH.parent}", "-pthread"], check=True, capture_output=True, text=True)
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.strip() == "fine", (run.returncode, run.stderr)
