"""The scratch of passes of more than 8 rows: B operands, and behind them room for partial sums, which the kernels read and write 16 bytes at a
time.  Nothing but the size of the first part keeps the second aligned."""
from __future__ import annotations

import random
import subprocess

import pytest

from vinf_3080ti_b200 import build

MAIN = """
#include "vqm_kernels.h"
#include <cstdio>
#include <cstdlib>
int main(int argc, char **argv) {
    size_t present = 0;
    for (int i = 1; i < argc; ++i) {
        present = vqm::tc_grown_split_bytes(std::strtoull(argv[i], nullptr, 10), present);
        std::printf("%zu\\n", present);
    }
    for (int sms = 1; sms <= 160; ++sms)
        if (vqm::tc_partial_count_bytes(sms) % 16 != 0 || vqm::kTcPartialAlign % 16 != 0) return 1;
}
"""


@pytest.fixture(scope="module")
def grown(tmp_path_factory):
    folder = tmp_path_factory.mktemp("split_scratch")
    source, program = folder / "sizes.cu", folder / "sizes"
    source.write_text(MAIN)
    subprocess.run([build._nvcc(), "-std=c++17", "-I", str(build.CSRC), str(source), "-o", str(program)], check=True)

    def run(needs):
        done = subprocess.run([str(program), *map(str, needs)], check=True, capture_output=True, text=True)
        return [int(line) for line in done.stdout.split()]

    return run


STEP = 42336  # bytes of Q4_K per 256 columns, 24 rows


@pytest.mark.parametrize("needs", [
    [1], [4 << 20], [(4 << 20) + 1],
    [STEP * ((cols + 255) // 256) for cols in (28928, 38400, 51200, 70000, 100000)],  # each outgrows the one before by less than half
    *([random.Random(seed).randrange(1, 1 << 26) for _ in range(12)] for seed in range(8)),
], ids=lambda needs: f"{len(needs)}-{needs[0]}")
def test_the_room_behind_the_operands_stays_aligned(grown, needs):
    wanted = []
    for need in needs:  # the runtime asks only for more
        if not wanted or need > grown(wanted)[-1]:
            wanted.append(need)
    sizes = grown(wanted)
    for i, (need, size) in enumerate(zip(wanted, sizes)):
        assert size >= need and size >= 4 << 20
        assert size % 256 == 0, sizes
        if i > 0:
            assert size >= sizes[i - 1] * 3 // 2 and sum(sizes[:i]) <= 2 * size
