"""The CTA bin with more pairs than it has resident CTAs."""
import numpy as np
import pytest

import canu_gb300 as oic
pytestmark = pytest.mark.gpu


def noisy(r, g, err):
    """A copy of g with substitutions, insertions and deletions, a third each."""
    x = r.random(len(g))
    out = np.where(x < err / 3, (g + r.integers(1, 4, len(g))) % 4, g)
    count = 1 + (x >= 2 * err / 3).astype(int) * (x < err) - (x >= err / 3).astype(int) * (x < 2 * err / 3)
    rid = np.repeat(np.arange(len(g)), count)
    out = out[rid]
    extra = np.flatnonzero(rid[1:] == rid[:-1]) + 1
    out[extra] = r.integers(0, 4, len(extra))
    return np.frombuffer(b"ACGT", np.uint8)[out].tobytes()


def pairs_of_reads(r, n, length, err):
    """n pairs of reads, each pair of a template of its own."""
    seqs = []
    for _ in range(n):
        g = r.integers(0, 4, length)
        seqs += [noisy(r, g, err), noisy(r, g, err)]
    return seqs


def run(seqs, reps=1, **tuning):
    off = np.cumsum([0] + [len(x) for x in seqs])
    with oic.Overlapper(oic.default_params(kmerLen=22, hashBits=20, maxErate=0.12, minOlapLen=300)) as ov:
        ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
        ov.set_tuning(**tuning)
        ms = []
        for _ in range(reps):
            ov.clear()
            ov.run()
            ms.append(ov.stats()["msWide"])
        return oic.sort_records(ov.overlaps()), ov.stats(), min(ms)


@pytest.fixture(scope="module")
def reads():
    r = np.random.default_rng(21)
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # One long pair more than there are SMs, and short ones that keep every SM busy about as
    # long as a long pair takes.
    return sms, pairs_of_reads(r, sms + 1, 7000, 0.05) + pairs_of_reads(r, 2500, 900, 0.05)


def test_records_do_not_depend_on_the_bin(reads, built):
    sms, seqs = reads
    warps, sw, _ = run(seqs)
    ctas, sc, _ = run(seqs, forceWide=1)
    assert sc["pairsWide"] > 2 * 2 * sms and len(ctas) > 2500
    assert np.array_equal(warps, ctas)
    for k in ("kmerHitsWithoutOlap", "kmerHitsWithOlap", "totalOverlaps", "containedOverlaps", "dovetailOverlaps"):
        assert sw[k] == sc[k], k


def test_longest_pairs_start_first_whatever_the_number_of_ctas(reads, built):
    """CTAs that wait for an SM hold no pair meanwhile: three CTAs for each SM take no longer
    than one (a long pair dealt to a waiting CTA starts when the short ones are done: half as
    long again)."""
    sms, seqs = reads
    _, _, one = run(seqs, 4, forceWide=1, wideCtas=sms)
    _, _, three = run(seqs, 4, forceWide=1, wideCtas=3 * sms)
    assert three < 1.15 * one, (one, three)


@pytest.mark.parametrize("tuning,per_sm", [({}, 1), ({"wideThreads": 256}, 2), ({"wideThreads": 64}, 2),
                                           ({"wideThreads": 256, "wideBandW": 25600}, 1)])
def test_default_ctas_are_those_the_sms_hold(tuning, per_sm, built):
    """No CTA of the default grid waits for an SM with its arena, rows and headers idle:
    128 registers a thread let one CTA of 512 threads, or two of 256, live on an SM, and
    200 KB of rows one."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    with oic.Overlapper(oic.default_params(kmerLen=22)) as ov:
        ov.set_tuning(**tuning)
        assert ov.tuning()["wideCtas"] == per_sm * sms


@pytest.mark.parametrize("graph", [0, 1])
def test_reruns_leave_no_counts_behind(graph, built):
    """Pairs whose extension does not fit a CTA's arena are discarded and run again in the
    large one: cells, rows and slide bases are those of a run whose arenas are large enough."""
    r = np.random.default_rng(23)
    seqs = pairs_of_reads(r, 3, 30000, 0.05) + pairs_of_reads(r, 20, 2000, 0.05)
    small, ss, _ = run(seqs, forceWide=1, noGraph=1 - graph, wideArena=1 << 20)
    large, sl, _ = run(seqs, forceWide=1, noGraph=1 - graph)
    assert ss["pairsWide"] > sl["pairsWide"]          # pairs were run again
    assert len(large) == 23 and np.array_equal(small, large)
    for k in ("dpCells", "dpRows", "extensions", "slideBases"):
        assert ss[k] == sl[k], (k, ss[k], sl[k])
