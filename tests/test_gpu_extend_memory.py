"""Batched extensions when there is no device memory for the CTA kernel's arenas."""
import numpy as np
import pytest

import canu_gb300 as oic
from test_gpu_rows import noisy

pytestmark = pytest.mark.gpu


def test_wide_bands_without_memory_for_the_cta_arenas(built):
    """A small batch hands bands wider than the shared-memory rows to the CTA kernel.  With
    arenas that no device holds (304 of 8 GB), the warps take them in HBM rows, and the
    results and the work counted are those of a batch that runs there anyway."""
    r = np.random.default_rng(22)
    pairs = noisy(r, 4, 16000, 0.02)
    seqs, prob = [], []
    for i, (s, t, ms, mt) in enumerate(pairs):
        seqs += [s.encode(), t.encode()]
        prob.append((2 * i + 1, 0, 2 * i + 2, ms, mt, 22))
    off = np.cumsum([0] + [len(x) for x in seqs])
    a = np.array(prob)
    got, cells = [], []
    for tuning, n in (({}, 1), ({"wideArena": 0x7fff0000, "wideCtas": 304}, 1), ({}, 400)):
        with oic.Overlapper(oic.default_params(kmerLen=22, maxErate=0.12)) as ov:
            ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
            ov.set_tuning(**tuning)
            b = np.tile(a, (n, 1))                 # 1,600 problems: more than eight per SM
            got.append([x[:len(a)] for x in ov.extend_batch(*[b[:, j] for j in range(6)])])
            cells.append(ov.stats()["dpCells"] / n)
    for other in got[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(got[0], other))
    assert (got[0][1] == 3).all()
    assert cells[1] == cells[2] < cells[0]         # the first batch's one-warp pass ran in vain
