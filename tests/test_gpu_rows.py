"""The one-warp DP where it can go wrong, against the oracle: slides that end around the 32-
and 1024-base steps, bands around the 32- and 64-diagonal chunks and past the shared-memory
rows, reads with N, both directions; and a pair whose match nodes keep helper warps busy."""
import ctypes

import numpy as np
import pytest

import canu_gb300 as oic
from test_gpu_edges import mutate, rand_seq, run_both
from test_gpu_extend import port_aligner

pytestmark = pytest.mark.gpu

K = 22
COMP = bytes.maketrans(b"acgtn", b"tgcan")


def slides(r):
    """Reads that agree over runs of given lengths, each ended by one error, on both sides of
    an exact seed in the middle."""
    pairs = []
    for run in (1, 31, 32, 33, 63, 64, 65, 96, 1023, 1024, 1025, 1055, 1056, 1057, 2048, 2081):
        for kind in "sid":
            left, seed, right = rand_seq(r, 2 * run + 40), rand_seq(r, K), rand_seq(r, 2 * run + 40)
            other = []
            for side, at in ((left, len(left) - 1 - run), (right, run)):
                c = side[at]
                new = {"s": "ACGT"[("ACGT".index(c) + 1) % 4], "i": c + "ACGT"[("ACGT".index(c) + 2) % 4], "d": ""}[kind]
                other.append(side[:at] + new + side[at + 1:])
            pairs.append((left + seed + right, other[0] + seed + other[1], len(left), len(other[0])))
    return pairs


def noisy(r, n, length, err, with_n=False):
    pairs = []
    for i in range(n):
        left, seed, right = rand_seq(r, length), rand_seq(r, K), rand_seq(r, length // 2 + 37 * i)
        a, b = mutate(r, left, err / 2), mutate(r, right, err / 2)
        c, d = mutate(r, left, err / 2), mutate(r, right, err / 2)
        if with_n:
            a = "".join("N" if r.random() < 0.01 else x for x in a)
            d = "".join("N" if r.random() < 0.01 else x for x in d)
        pairs.append((a + seed + b, c + seed + d, len(a), len(c)))
    return pairs


def unrelated(r):
    return [(rand_seq(r, 900), rand_seq(r, 1100), 400 + i, 500 - i) for i in range(8)]


@pytest.mark.parametrize("name,erate,partial", [("slides", 0.06, 0), ("slides", 0.01, 1), ("narrow", 0.02, 0),
                                                ("mid", 0.06, 0), ("wide", 0.12, 0), ("wide", 0.12, 1), ("n", 0.06, 0),
                                                ("unrelated", 0.12, 0)])
def test_row_loop_edges_match_oracle(name, erate, partial, built, oracle):
    r = np.random.default_rng(11)
    pairs = {"slides": lambda: slides(r), "narrow": lambda: noisy(r, 6, 3000, 0.012), "mid": lambda: noisy(r, 6, 2500, 0.03),
             # 2 % error under a 12 % limit: the band passes 508 diagonals after some 400 rows
             "wide": lambda: noisy(r, 2, 26000, 0.02), "n": lambda: noisy(r, 6, 2000, 0.03, True),
             "unrelated": lambda: unrelated(r)}[name]()
    seqs, prob = [], []
    for i, (s, t, ms, mt) in enumerate(pairs):
        rev = i % 2
        stored = s.encode().lower()
        seqs += [stored[::-1].translate(COMP) if rev else stored, t.encode().lower()]
        prob.append((2 * i + 1, rev, 2 * i + 2, ms, mt, K))
    off = np.cumsum([0] + [len(x) for x in seqs])
    erate = float(np.float32(erate))
    with oic.Overlapper(oic.default_params(kmerLen=K, maxErate=erate, partial=partial)) as ov:
        ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
        a = np.array(prob)
        out, kind, dl = ov.extend_batch(*[a[:, j] for j in range(6)])
    plib = ctypes.CDLL(oracle["lib"])
    al = port_aligner(plib, erate, 1.0, partial)
    for i, (s, t, ms, mt) in enumerate(pairs):
        o, n = np.zeros(5, dtype=np.int32), ctypes.c_int32()
        k = plib.oic_port_extend(al, s.encode().lower(), len(s), t.encode().lower(), len(t), ms, mt, K, o.ctypes.data, None,
                                 ctypes.byref(n), None, None)
        assert k == kind[i] and (o == out[i]).all() and n.value == dl[i], (i, k, o, n.value, kind[i], out[i], dl[i])
    plib.oic_port_aligner_free(al)


@pytest.mark.parametrize("extra", [[], ["-m"], ["-partial"]])
def test_few_pairs_with_many_nodes(extra, built, oracle, tmp_path):
    """Three reads, hundreds of match nodes a pair: every other warp of the owners' CTAs
    helps, and the records and counts are those of one extension after another."""
    r = np.random.default_rng(12)
    g = rand_seq(r, 16000)
    seqs = [mutate(r, g, 0.015), mutate(r, g[2000:], 0.015), mutate(r, g[:13000], 0.015)]
    rec = run_both(built, oracle, tmp_path, seqs, ["-t", "2", "-k", "22", "--hashbits", "16", "--maxerate", "0.06",
                                                   "--minlength", "500"] + extra)
    assert len(rec) >= 3


@pytest.mark.parametrize("err,erate,with_n", [(0.0055, 0.01, False), (0.0055, 0.01, True), (0.011, 0.02, False),
                                              (0.024, 0.045, False), (0.004, 0.06, False)])
def test_hopeless_groups_keep_records(err, erate, with_n, built):
    """Read pairs just above and below the error limit, and pairs that share a repeat only:
    the one-warp DP, which drops groups of match nodes it shows to have no overlap, against
    the CTA DP, which extends each of them."""
    r = np.random.default_rng(13)
    rep = rand_seq(r, 3000)
    g = rand_seq(r, 9000) + rep + rand_seq(r, 12000) + mutate(r, rep, 0.01) + rand_seq(r, 9000) + mutate(r, rep, 0.02)
    seqs = []
    for _ in range(45):
        n = int(r.integers(2500, 9000))
        p = int(r.integers(0, len(g) - n))
        s = mutate(r, g[p:p + n], err)
        if with_n:
            s = "".join("N" if r.random() < 0.0005 else c for c in s)
        seqs.append((s if r.random() < 0.5 else s[::-1].translate(str.maketrans("ACGT", "TGCA"))).encode())
    off = np.cumsum([0] + [len(x) for x in seqs])
    got = []
    for wide in (0, 1):
        with oic.Overlapper(oic.default_params(kmerLen=K, hashBits=18, maxErate=erate, minOlapLen=500)) as ov:
            ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
            ov.set_tuning(forceWide=wide)
            ov.run()
            got.append((oic.sort_records(ov.overlaps()), ov.stats()))
    (a, sa), (b, sb) = got
    assert a.shape == b.shape and (a == b).all()
    for k in ("kmerHitsWithoutOlap", "kmerHitsWithOlap", "kmerHitsSkipped", "multiOverlap", "totalOverlaps",
              "containedOverlaps", "dovetailOverlaps", "seeds", "candidatePairs", "nodes"):
        assert sa[k] == sb[k], k
    if erate <= 0.02:
        assert sa["extensions"] < sb["extensions"]   # groups were dropped


@pytest.mark.parametrize("erate", [0.01, 0.02])
def test_collected_pairs_count_the_reference_extensions(erate, built):
    """The extensions and the first hit of a collected pair do not depend on which of its
    match nodes were shown to have no overlap without extending them."""
    r = np.random.default_rng(14)
    rep = rand_seq(r, 2500)
    g = rand_seq(r, 6000) + rep + rand_seq(r, 9000) + mutate(r, rep, 0.01) + rand_seq(r, 6000)
    seqs = []
    for _ in range(40):
        n = int(r.integers(2500, 8000))
        p = int(r.integers(0, len(g) - n))
        seqs.append(mutate(r, g[p:p + n], 0.55 * erate).encode())
    off = np.cumsum([0] + [len(x) for x in seqs])
    got = []
    for wide in (0, 1):
        with oic.Overlapper(oic.default_params(kmerLen=K, hashBits=18, maxErate=erate, minOlapLen=500)) as ov:
            ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
            ov.set_tuning(forceWide=wide)
            ov.collect_pairs(1)
            ov.run()
            info = ov.pairs()[0]
            got.append((info[np.lexsort((info["flags"], info["bID"], info["aID"]))], ov.stats()["extensions"]))
    (a, na), (b, nb) = got
    assert na < nb   # groups were dropped
    for k in ("aID", "bID", "flags", "nodes", "overlaps", "extensions", "firstHit"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("erate", [0.12])
def test_wide_bands_by_warps_and_by_ctas(erate, built):
    """Bands wider than the shared-memory rows: a small batch hands them to the CTA kernel, a
    large one keeps them on a warp, or on smaller CTAs when these are asked for; the results
    are the same."""
    r = np.random.default_rng(15)
    seqs, prob = [], []
    for i in range(9):
        g = rand_seq(r, 9000 + 1500 * i)
        seqs += [mutate(r, g, 0.05).encode(), mutate(r, g, 0.05).encode()]
        anchor = next((p, q) for p in range(2000, 8000) for q in [seqs[-1].find(seqs[-2][p:p + K])] if q >= 0)
        prob.append((2 * i + 1, 0, 2 * i + 2, anchor[0], anchor[1], K))
    off = np.cumsum([0] + [len(x) for x in seqs])
    with oic.Overlapper(oic.default_params(kmerLen=K, maxErate=erate)) as ov:
        ov.set_reads(np.ones(len(seqs)), [len(x) for x in seqs], off[:-1], np.frombuffer(b"".join(seqs), np.uint8))
        a = np.array(prob)
        small = ov.extend_batch(*[a[:, j] for j in range(6)])
        b = np.tile(a, (300, 1))                 # 2,700 problems: more than eight per SM
        large = ov.extend_batch(*[b[:, j] for j in range(6)])
        ov.set_tuning(forceWide=1)
        forced = ov.extend_batch(*[b[:, j] for j in range(6)])
    assert (small[1] == 3).any()                 # some reach both ends
    for s, l, f in zip(small, large, forced):
        want = np.tile(s, (300,) + (1,) * (s.ndim - 1))
        assert (want == l).all() and (want == f).all()
