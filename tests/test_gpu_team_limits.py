"""The bounded waits of the one-warp DP's teams, made to run out: the library's pair kernels
compiled with short limits give the records and counts of the ordinary ones."""
import os
import subprocess
import sys

import numpy as np
import pytest

import canu_gb300 as oic
from canu_gb300 import build
from test_gpu_edges import mutate, rand_seq

pytestmark = pytest.mark.gpu

RUN = """
import sys
import numpy as np
import canu_gb300 as oic
oic.LIB_PATH, data, out = sys.argv[1:]
z = np.load(data)
res = []
for collect in (0, 1):
    with oic.Overlapper(oic.default_params(kmerLen=22, hashBits=18, maxErate=float(z["erate"]), minOlapLen=500)) as ov:
        ov.set_reads(np.ones(len(z["len"])), z["len"], z["off"], z["bases"])
        ov.collect_pairs(collect)
        ov.run()
        s = ov.stats()
        res.append((oic.sort_records(ov.overlaps()), [s[k] for k in
                    ("kmerHitsWithOlap", "kmerHitsWithoutOlap", "multiOverlap", "totalOverlaps", "dovetailOverlaps",
                     "containedOverlaps", "candidatePairs", "pairsWide")]))
np.savez(out, a=res[0][0], b=res[1][0], sa=res[0][1], sb=res[1][1])
"""


@pytest.fixture(scope="module")
def run(built, tmp_path_factory):
    d = tmp_path_factory.mktemp("team")
    r = np.random.default_rng(25)
    rep = rand_seq(r, 2500)
    g = rand_seq(r, 7000) + rep + rand_seq(r, 7000) + mutate(r, rep, 0.01) + rand_seq(r, 5000)
    seqs = []
    for _ in range(36):
        n = int(r.integers(4000, 12000))
        p = int(r.integers(0, len(g) - n))
        seqs.append(mutate(r, g[p:p + n], 0.015).encode())
    np.savez(d / "reads.npz", len=[len(s) for s in seqs], off=np.cumsum([0] + [len(s) for s in seqs])[:-1],
             bases=np.frombuffer(b"".join(seqs), np.uint8), erate=0.045)

    def go(lib, name):
        out = str(d / (name + ".npz"))
        p = subprocess.run([sys.executable, "-c", RUN, lib, str(d / "reads.npz"), out], cwd=os.path.dirname(build.HERE),
                           stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
        assert p.returncode == 0, p.stdout[-2000:]
        return np.load(out)

    def variant(name, defines):
        obj, lib = str(d / (name + ".o")), str(d / (name + ".so"))
        build._run([build.nvcc()] + build.ARCH + build.NVFLAGS + defines + ["-c", os.path.join(build.CSRC, "oic_pairs.cu"),
                                                                            "-o", obj])
        others = [os.path.join(build.OUT, os.path.splitext(s)[0] + ".o") for s in build.CU_SOURCES + build.HOST_SOURCES
                  if s != "oic_pairs.cu"]
        build._run([build.nvcc()] + build.ARCH + ["-shared", "-o", lib, obj] + others + ["-lcudart"])
        return go(lib, name)
    return lambda: go(oic.LIB_PATH, "ordinary"), variant


@pytest.mark.parametrize("name,defines", [("locks", ["-DOIC_LOCK_TRIES=0"]), ("waits", ["-DOIC_WAIT_TRIES=3"]),
                                          ("both", ["-DOIC_LOCK_TRIES=1", "-DOIC_WAIT_TRIES=40"])])
def test_waits_that_run_out_change_no_record(name, defines, run):
    ordinary, variant = run
    want, got = ordinary(), variant(name, defines)
    assert len(want["a"]) > 100
    for k in ("a", "b"):
        assert np.array_equal(want[k], got[k]), k
    for k in ("sa", "sb"):
        assert np.array_equal(want[k][:-1], got[k][:-1]), k
    assert want["sa"][-1] == 0
    if name == "locks":
        assert got["sa"][-1] > 0      # helpers kept an owner from its pair, which went to the CTA bin
