"""Order of the tiled posterior decoding, on the host: the kernel's own schedule
(messi_gb300/csrc/decode_schedule.h, compiled here) is walked for every tile with
a vector clock per CTA, so that a tile counts as written only where a flag that
the CTA has waited for, or its own program order, says so.  However late any CTA
is, no tile may be read before that, and no wait may be for a flag that is raised
later."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "messi_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "decode_schedule.h"
int main(int argc, char** argv)
{
    const int NB = std::atoi(argv[1]);
    for (int D = 1; D < NB; D++)
        for (int I = 0; I + D < NB; I++) {
            const messi::DecodeWait e = messi::decode_early_wait(I, D), l = messi::decode_late_wait(I, D);
            std::printf("%d %d %d %d %d %d %d\n", D, I, messi::decode_early_first(I), e.block, e.diagonals, l.block,
                        l.diagonals);
        }
}
"""


@pytest.fixture(scope="module")
def schedule(tmp_path_factory):
    d = tmp_path_factory.mktemp("decode_schedule")
    (d / "walk.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, str(d / "walk.cpp"), "-o", str(d / "walk")], check=True)

    def rows(nb):
        out = subprocess.run([str(d / "walk"), str(nb)], check=True, capture_output=True, text=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return rows


def walk(rows, nb, grid):
    """Reads of unfinished tiles, as (D, I, row block, column block, stage), and
    waits for flags that are not raised by an earlier diagonal."""
    known = [np.zeros(nb, dtype=int) for _ in range(grid)]  # per CTA: diagonals known to be finished of each block
    raised = {}
    for i in range(nb):  # the diagonal tiles, each CTA's blocks in order
        c = known[i % grid]
        c[i] = 1
        raised[i, 1] = c.copy()
    unordered, stuck = [], []

    def wait(c, block, diagonals):
        if diagonals <= 0:
            return
        if (block, diagonals) not in raised:
            stuck.append((block, diagonals))
        else:
            np.maximum(c, raised[block, diagonals], out=c)

    for D, i, first, eb, en, lb, ln in rows:
        c, j = known[i % grid], i + D

        def read(r, col, stage):
            if r <= col and c[r] < col - r + 1:
                unordered.append((D, i, r, col, stage))

        wait(c, eb, en)
        for r in range(first, j):
            read(r, j, "early")
        wait(c, lb, ln)
        for r in range(i + 1, min(first, j)):
            read(r, j, "late")
        for r, col in ((j, j), (i + 1, j), (i + 1, j - 1), (i, j - 1)):
            read(r, col, "late")
        c[i] = D + 1
        raised[i, D + 1] = c.copy()
    return unordered, stuck


@pytest.mark.parametrize("nb", [2, 3, 4, 5, 8, 17, 63, 154])
def test_no_tile_is_read_before_it_is_written(schedule, nb):
    rows = schedule(nb)
    assert len(rows) == nb * (nb - 1) // 2
    for grid in sorted({1, 2, 3, 4, 5, 7, nb - 1, nb}):
        if grid > nb:
            continue
        unordered, stuck = walk(rows, nb, grid)
        assert not stuck, (grid, stuck[:3])
        assert not unordered, (grid, len(unordered), unordered[:3])
