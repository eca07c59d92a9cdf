"""Device memory of the overlap-store record pass (CPU: its layout, compiled for the host)."""
import os
import subprocess

import pytest

from conftest import ROOT

NAMES = ["in", "keys", "keep", "pos", "rec", "k2", "k3", "idx", "idx2", "scr", "cnt", "a", "aOff", "out", "bytes"]


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("layout") / "layout")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "canu_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "store_layout_main.cpp"), "-o", exe], check=True)

    def run(n, max_id, scr):
        out = subprocess.run([exe], input=f"{n} {max_id} {scr}\n", stdout=subprocess.PIPE, text=True, check=True).stdout
        return dict(zip(NAMES, map(int, out.split())))
    return run


@pytest.mark.parametrize("n", [0, 1, 2, 31, 32, 33, 1000, 1_500_007, 0x7fffffff])
@pytest.mark.parametrize("max_id", [1, 60_013, 0xffffffff])
def test_arrays_do_not_overlap_and_no_output_is_held_that_may_not_come(n, max_id, layout):
    scr = 4096 + n // 16
    size = {"in": 24 * n, "keys": 16 * n, "keep": 4 * (2 * n + 1), "pos": 4 * (2 * n + 1), "rec": 48 * n, "k2": 16 * n,
            "k3": 16 * n, "idx": 8 * n, "idx2": 8 * n, "scr": scr, "cnt": 80, "a": 4 * (max_id + 2),
            "aOff": 4 * (max_id + 2)}
    at = layout(n, max_id, scr)
    end = 0
    for k in sorted(size, key=lambda k: (at[k], size[k])):
        assert at[k] % 256 == 0 and at[k] >= end, k
        end = at[k] + size[k]
    assert at["bytes"] >= end
    # The output lies over what is dead by then (the records as read, the keys and flags of
    # all copies) and does not reach the arrays that it is gathered from.
    live = min(at[k] for k in ("rec", "k2", "k3", "idx", "idx2", "scr", "cnt", "a", "aOff"))
    assert at["out"] % 256 == 0 and at["out"] + 48 * n <= live
    # 152 bytes a record, scratch, and the two counters per read: nothing for copies that the
    # error rate may drop.
    assert at["bytes"] <= 152 * n + scr + 8 * max_id + 13 * 256 + 200
