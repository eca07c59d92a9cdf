"""Positions in a hash block's occurrence array as the seed kernel computes them (CPU: the
kernel's own header, compiled for the host)."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def positions(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("occ") / "occurrences")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "canu_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "occurrences_main.cpp"), "-o", exe], check=True)

    def run(queries):
        text = "".join(" ".join(map(str, q)) + "\n" for q in queries)
        out = subprocess.run([exe], input=text, stdout=subprocess.PIPE, text=True, check=True, timeout=60).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


@pytest.mark.parametrize("base", [0, (1 << 31) - 40, 1 << 31, 3_000_000_000, (1 << 32) - 2 - 5000])
def test_search_finds_the_first_partner_anywhere_in_the_array(base, positions):
    """Runs of 0 to 5,000 occurrences from `base` on, past 2^31 and up to the last position a
    block may have: the position found is the first of a string >= from, and nothing outside
    the run is read."""
    r = np.random.default_rng(19)
    queries, want = [], []
    for length in (0, 1, 2, 3, 64, 65, 1000, 4999, 5000):
        for div in (1, 7, 100_000):
            start = base + int(r.integers(0, 5000 - length + 1))
            end = start + length
            for from_ in {0, start // div, (start + length // 2) // div, (start + length // 2) // div + 1, end // div + 1}:
                queries.append(("s", start, end, from_, div))
                want.append((min(max(start, from_ * div), end), 0))
    assert positions(queries) == want


def test_seeds_of_256_offsets_do_not_wrap(positions):
    """The 32-bit sum of the seeds of 256 ref offsets is the 64-bit one for every run up to the
    longest that the widest configuration can hold; longer runs are refused, each of them
    (16,777,216 seeds an offset made the sum 0, and a little more a small number)."""
    cap = 1 << 22
    counts = [0, 1, cap - 1, cap, cap + 1, (1 << 24) - 1, 1 << 24, (1 << 24) + 1, (1 << 31) - 1]
    got = positions([("o", 1000, 1000 + n, 0, 7) for n in counts])
    assert got == [(256 * n, 0) if n < cap else (0, 256) for n in counts]
    # Only the occurrences from the first qualifying string on count: the last 70 of 4 strings.
    assert positions([("o", 0, 280, 3, 70), ("o", 0, 280, 4, 70)]) == [(256 * 70, 0), (0, 0)]
