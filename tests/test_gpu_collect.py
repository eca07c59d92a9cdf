"""Collected pairs: their extensions and cells are those of one extension after another, and
collecting does not change the work that the run reports."""
import numpy as np
import pytest

import canu_gb300 as oic
from test_gpu_edges import mutate, rand_seq

pytestmark = pytest.mark.gpu

WORK = ("dpCells", "dpRows", "slideBases", "extensions", "totalOverlaps", "kmerHitsWithOlap", "kmerHitsWithoutOlap")


@pytest.mark.parametrize("erate,with_n", [(0.01, False), (0.02, False), (0.01, True)])
def test_cells_of_collected_pairs_are_those_of_their_extensions(erate, with_n, built):
    """The one-warp DP settles groups of match nodes together; the CTA DP extends each node.
    A collected pair's cells and extensions, from which the trainer takes the cost of an
    extension, do not depend on which of them ran."""
    r = np.random.default_rng(24)
    rep = rand_seq(r, 2500)
    g = rand_seq(r, 6000) + rep + rand_seq(r, 9000) + mutate(r, rep, 0.01) + rand_seq(r, 6000)
    seqs = []
    for _ in range(40):
        n = int(r.integers(2500, 8000))
        p = int(r.integers(0, len(g) - n))
        s = mutate(r, g[p:p + n], 0.55 * erate)
        seqs.append("".join("N" if with_n and r.random() < 0.0005 else c for c in s).encode())
    off = np.cumsum([0] + [len(x) for x in seqs])

    def run(collect, wide):
        with oic.Overlapper(oic.default_params(kmerLen=22, hashBits=18, maxErate=erate, minOlapLen=500)) as ov:
            ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
            ov.set_tuning(forceWide=wide)
            ov.collect_pairs(collect)
            ov.run()
            info = ov.pairs()[0]
            return (info[np.lexsort((info["flags"], info["bID"], info["aID"]))], ov.stats(),
                    oic.sort_records(ov.overlaps()))

    plain, sp, rp = run(0, 0)
    a, sa, ra = run(1, 0)
    b, sb, rb = run(1, 1)
    assert len(plain) == 0 and len(a) == len(b) > 100
    assert np.array_equal(rp, ra) and np.array_equal(rp, rb)
    assert sa["extensions"] < sb["extensions"]      # groups were settled together
    assert [sp[k] for k in WORK] == [sa[k] for k in WORK]
    for k in ("aID", "bID", "flags", "nodes", "overlaps", "extensions", "firstHit", "cells", "cellsFirst"):
        assert np.array_equal(a[k], b[k]), k
    assert int(b["cells"].sum()) == sb["dpCells"] and int(b["extensions"].sum()) == sb["extensions"]
