"""The seed replay at its edges, against the oracle: more seeds per 256 offsets than the
buffer holds, several occurrences of one partner per offset, occurrence runs past the scan
limit, more partners than a strand's pair table holds, reads around one step of offsets,
reads with N."""
import numpy as np
import pytest

from test_gpu_edges import mutate, rand_seq, run_both

pytestmark = pytest.mark.gpu

ARGS = ["-t", "2", "-k", "22", "--hashbits", "18", "--maxerate", "0.06", "--minlength", "200"]


def tandem(r):
    unit = rand_seq(r, 37)
    return [mutate(r, rand_seq(r, 150) + unit * 20 + rand_seq(r, 150 + 7 * i), 0.01) for i in range(14)], ARGS


def shared_repeat(r):
    rep = rand_seq(r, 700)
    return [rand_seq(r, 90 + 3 * i) + mutate(r, rep, 0.004) + rand_seq(r, 200) for i in range(90)], ARGS


def many_partners(r):
    g = rand_seq(r, 420)
    seqs = [mutate(r, g, 0.003) for _ in range(2300)]
    return seqs, ARGS + ["-h", "1-2300", "-r", "1-4"]


def step_edges(r):
    g = rand_seq(r, 3000)
    # k-mer offsets (length - 21) around multiples of 256, a fixed start
    return [mutate(r, g[:n + 21], 0.002)[:n + 21] for n in (255, 256, 257, 511, 512, 513, 768, 1025, 1279)], ARGS


def with_n(r):
    g = rand_seq(r, 2500)
    return ["".join("N" if r.random() < 0.01 else c for c in mutate(r, g[40 * i:], 0.01)) for i in range(12)], ARGS


@pytest.mark.parametrize("make", [tandem, shared_repeat, many_partners, step_edges, with_n])
def test_seed_replay_matches_oracle(make, built, oracle, tmp_path):
    seqs, args = make(np.random.default_rng(17))
    run_both(built, oracle, tmp_path, seqs, args)   # records, .oc and stats (the k-mer hit counts) are equal
