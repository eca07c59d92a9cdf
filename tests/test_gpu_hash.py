"""The hash block around its entry limit: a block whose k-mers cannot meet the limit is built
without counting each string's new ones; the last read, the table and the records are those
of the counted block."""
import numpy as np
import pytest

import canu_gb300 as oic
from test_gpu_edges import COMP, mutate, rand_seq

pytestmark = pytest.mark.gpu
K, BITS, PER_BUCKET = 22, 16, 21


def reads(r, unique):
    if unique:
        seqs = [rand_seq(r, n) for n in (900, 1300, 801, 1000)]
    else:
        g = rand_seq(r, 6000)
        seqs = [mutate(r, g[p:p + 2500], 0.01) for p in r.integers(0, 3500, 24)]
        seqs = [s if i % 3 else s[::-1].translate(COMP) for i, s in enumerate(seqs)]
        seqs[5] = seqs[5][:700] + "N" + seqs[5][701:]
    return seqs + [rand_seq(r, 300), rand_seq(r, 250)]   # shorter than an overlap: no k-mers


def last_read(seqs, limit, min_len):
    seen = set()
    for i, s in enumerate(seqs):
        if len(seen) >= limit:
            return i
        if len(s) >= min_len:
            seen |= {s[o:o + K] for o in range(len(s) - K + 1) if "N" not in s[o:o + K]}
    return len(seqs)


@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("past", [-700, -1, 0, 1, 700])
def test_block_at_its_entry_limit(unique, past, built):
    seqs = reads(np.random.default_rng(3), unique)
    flat = sum(len(s) - K + 1 for s in seqs if len(s) >= 500)
    limit = flat + past
    off = np.cumsum([0] + [len(s) for s in seqs])
    got = []
    for lim in (limit, 10 * flat):
        p = oic.default_params(kmerLen=K, hashBits=BITS, maxErate=0.06, minOlapLen=500,
                               maxHashLoad=(lim + 0.5) / ((1 << BITS) * PER_BUCKET))
        with oic.Overlapper(p) as ov:
            ov.set_reads(np.ones(len(seqs)), [len(s) for s in seqs], off[:-1],
                         np.frombuffer("".join(seqs).encode(), np.uint8))
            assert ov.load_hash_block(1, len(seqs)) == last_read(seqs, lim, 500)
            ov.run()
            got.append(oic.sort_records(ov.overlaps()))
    assert got[0].shape == got[1].shape and (got[0] == got[1]).all() and (unique or len(got[0]) > 20)
