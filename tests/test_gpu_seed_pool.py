"""A ref offset with more seeds than a strand's node pool holds (32,768 match nodes in the
first configuration): the strand is given up at once and runs in the wide one, and the
records and counts are the oracle's."""
import numpy as np
import pytest

from test_gpu_edges import mutate, rand_seq, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [16, 17])   # of one k-mer in each of 2,000 partners: 32,000 and 34,000 seeds
def test_one_offset_with_more_seeds_than_nodes(copies, built, oracle, tmp_path):
    r = np.random.default_rng(20)
    word = rand_seq(r, 22)
    g = rand_seq(r, 900)
    ref = g[:450] + word + g[450:]
    seqs = [ref, mutate(r, ref, 0.01)]
    seqs += ["".join(word + rand_seq(r, 9) for _ in range(copies)) for _ in range(2000)]
    rec = run_both(built, oracle, tmp_path, seqs, ["-t", "2", "-k", "22", "--hashbits", "18", "--maxerate", "0.06",
                                                   "--minlength", "300", "-r", "1-2"])
    assert len(rec) == 1
