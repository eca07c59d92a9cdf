"""The radix sort under the store build and the k-mer count at its edges: records around one
tile, ID widths around a digit, digits that are all equal, windows around a block's step,
more k-mers than the first count has room for."""
import numpy as np
import pytest

import canu_gb300 as oic
from test_gpu_store import check
from test_kmers import ko
from test_store_oracle import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 2047, 2048, 2049, 6143, 6145])   # two copies of each: tiles of 4,096
@pytest.mark.parametrize("max_id", [1, 3, 255, 256, 65535, 65536, 1 << 22])
def test_store_sort_at_tile_and_digit_edges(n, max_id, built):
    n = min(n, 40) if max_id < 255 else n   # one pair's records are ordered by one thread
    rec = synthetic(n, 50, seed=n)
    r = np.random.default_rng(n + max_id)
    rec[:, :2] = r.integers(max(1, max_id - 300), max_id + 1, size=(n, 2))   # top digits alike
    check(rec, max_id, 1.0)



@pytest.mark.parametrize("k,lens", [(22, (21, 22, 23, 1044, 1045, 1046, 2069)), (31, (31, 1054, 1055)), (11, (4106, 4107))])
def test_count_at_window_edges(k, lens, built):
    r = np.random.default_rng(k)
    reads = ["".join(r.choice(list("ACGT"), n)) for n in lens] * 2
    reads[0] = reads[0][:-1] + "N"
    check_count(reads, k, 2)


def test_count_past_the_first_room(built):
    r = np.random.default_rng(1)
    check_count(["".join(r.choice(list("ACGT"), 90000)) for _ in range(3)], 22, 1)   # 269,937 k-mers


def check_count(reads, k, min_count):
    data = [s.encode() for s in reads]
    off = np.cumsum([0] + [len(s) for s in data])[:-1].astype(np.uint64)
    with oic.Overlapper(oic.default_params(kmerLen=k)) as ov:
        ov.set_reads(np.ones(len(data)), [len(s) for s in data], off, np.frombuffer(b"".join(data), dtype=np.uint8))
        strs, cnt = ov.count_kmers(1, len(data), min_count)
    ref_s, ref_c = ko.frequent(data, k, min_count)
    assert strs == ref_s and np.array_equal(cnt, ref_c)
