"""Performance cases of the GB300 overlapInCore engine: what a user of the library has it
do, at the sizes it is used at.

listed() names the cases, draw() makes more of the same ranges, prepare() builds what a
program holds before the call, run() is one pass through the public entry points, work()
the bytes and operations the pass cannot do without, exact() the 64-bit value of the
outputs that are floating-point numbers.

Read sets are drawn on the GPU from the seed alone with the shapes of the benchmark
workloads (canu_gb300/workloads.py): a random genome with dispersed repeats and tandem
arrays, read lengths by law, substitutions / insertions / deletions, both strands.

Kinds of case
  job     one overlap job: reads from host memory to the device, every hash block against
          the ref range, records home and in overlap-store order (the order canu's later
          stages need, and the only order two runs share)
  extend  a batch of seed extensions (Extend_Alignment) on a loaded read store
  kmers   the frequent-k-mer count that makes a job's skip list
  store   the record pass of the overlap-store build
  train   one optimizer step of the learned filter: forward, backward, Adam
"""
import math
import os

import numpy as np
import torch

import canu_gb300 as oic
from canu_gb300 import filter_train

K = 22
DEVICE = "cuda"
FILTER = os.path.join(os.path.dirname(os.path.abspath(oic.__file__)), "filter_c2.npz")


def _job(name, **kw):
    d = dict(name=name, kind="job", genome=1_000_000, coverage=20.0, law="lognormal", mean=8000, sd=3000, lo=1000,
             hi=30000, err=0.02, ins=1, dele=1, n_rate=0.0, copies=0, tandem=0.0, erate=0.06, minlen=500, bits=23,
             load=0.6, data=100_000_000, partial=0, multi=0, skip=0, filter=0, refs=0)
    d.update(kw)
    return d


def _hifi(name, **kw):
    d = dict(coverage=30.0, law="normal", mean=15000, sd=3000, err=0.005, tandem=0.02, erate=0.01, minlen=1000, bits=25,
             data=1_600_000_000, skip=1)
    d.update(kw)
    return _job(name, **d)


def listed():
    return [
        # The smallest call: a few dozen reads, as a bacterial test set or one bin of a
        # metagenome; latency of the whole chain of launches.
        _job("job_few_reads", genome=24_000, coverage=10.0, mean=4000, sd=1500, bits=18, data=10_000_000),
        # An ordinary job: 2 % reads of lognormal length at the reference's default error
        # rate, unique overlaps, one hash block, no skip list.
        _job("job_lognormal_2pct", genome=1_003_000, load=0.8),
        # The headline shape: HiFi reads with dispersed repeats, tandem arrays and the
        # skip list, at a tenth of its genome.
        _hifi("job_hifi_repeats", genome=5_000_000, copies=20),
        # The same reads through the learned candidate filter.
        _hifi("job_hifi_filtered", genome=5_000_000, copies=20, filter=1),
        # Noisy reads of heavy-tailed length at 12 % error rate: wide bands, many
        # extensions per pair.
        _job("job_noisy_pareto", genome=150_000, coverage=25.0, law="pareto", mean=0, sd=0, lo=500, hi=14_000, err=0.05,
             ins=2, dele=2, erate=0.12, bits=24, data=600_000_000),
        # Trimming's overlaps: -partial, every overlap of a pair kept (-m), reads with N,
        # a skip list, two hash blocks.
        _job("job_partial_multi", genome=250_001, coverage=16.0, mean=7000, sd=2500, err=0.015, n_rate=2e-4, copies=14,
             erate=0.045, bits=22, data=600_000, partial=1, multi=1, skip=1),
        # One job of a partitioned assembly: a whole hash block against a narrow ref
        # range, so that loading reads and building the block are most of it.
        _hifi("job_block_few_refs", genome=8_000_000, coverage=25.0, copies=32, refs=211),
        # Many ordinary seed extensions, both strands, ragged lengths.
        dict(name="extend_many", kind="extend", n=20_011, mean=7000, sd=2500, lo=600, hi=20000, err=0.01, ins=1, dele=1,
             erate=0.045),
        # A few long noisy ones, whose bands need the whole CTA.
        dict(name="extend_long", kind="extend", n=230, mean=60000, sd=15000, lo=20000, hi=100000, err=0.04, ins=2, dele=2,
             erate=0.12),
        # The skip list of a 30x read set: every canonical 22-mer seen 300 times or more.
        dict(name="kmer_count", kind="kmers", genome=4_000_000, coverage=30.0, mean=15000, sd=3000, err=0.005, copies=16,
             tandem=0.02, min_count=300),
        # Store build over the records of several jobs.
        dict(name="store_records", kind="store", n=1_500_007, reads=60_013, erate=0.045),
        # One training step of the filter network at the trainer's batch.
        dict(name="filter_train_step", kind="train", n=32768, pos=0.1),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["2pct", "2pct", "hifi", "hifi", "filter", "noisy", "partial", "slice", "many", "long", "kmers",
                       "store", "train"])
    if kind == "2pct":
        d = _job("", genome=_log(rng, 20_000, 1_500_000), coverage=round(rng.uniform(8, 25), 1),
                 mean=rng.randrange(3000, 10001), sd=rng.randrange(800, 3501), err=round(rng.uniform(0.008, 0.024), 4),
                 erate=rng.choice([0.045, 0.06]), bits=rng.choice([20, 22, 23]), multi=rng.choice([0, 0, 1]))
    elif kind in ("hifi", "filter"):
        g = _log(rng, 200_000, 4_800_000)
        d = _hifi("", genome=g, coverage=round(rng.uniform(15, 30), 1), mean=rng.randrange(10000, 18001),
                  sd=rng.randrange(1500, 3501), err=round(rng.uniform(0.002, 0.006), 4), copies=g // 250_000,
                  filter=int(kind == "filter"))
    elif kind == "noisy":
        d = _job("", genome=_log(rng, 20_000, 140_000), coverage=round(rng.uniform(10, 25), 1), law="pareto", mean=0, sd=0,
                 lo=500, hi=rng.randrange(5000, 13001), err=round(rng.uniform(0.03, 0.05), 4), ins=2, dele=2, erate=0.12,
                 bits=24, data=600_000_000)
    elif kind == "partial":
        g = _log(rng, 30_000, 250_000)
        d = _job("", genome=g, coverage=round(rng.uniform(8, 16), 1), mean=rng.randrange(3000, 8001),
                 sd=rng.randrange(800, 2501), err=round(rng.uniform(0.005, 0.015), 4), n_rate=rng.choice([0.0, 1e-4, 1e-3]),
                 copies=g // 15_000, erate=0.045, bits=22, data=rng.choice([300_000, 600_000, 100_000_000]), partial=1,
                 multi=rng.choice([0, 1]), skip=1)
    elif kind == "slice":
        g = _log(rng, 1_000_000, 8_000_000)
        d = _hifi("", genome=g, coverage=round(rng.uniform(15, 25), 1), copies=g // 250_000, refs=rng.randrange(17, 400))
    elif kind == "many":
        m = rng.randrange(1500, 9001)
        d = dict(kind="extend", n=_log(rng, 37, 20_000), mean=m, sd=m // 3, lo=400, hi=3 * m,
                 err=round(rng.uniform(0.003, 0.02), 4), ins=1, dele=1, erate=rng.choice([0.02, 0.045, 0.06]))
    elif kind == "long":
        m = rng.randrange(25000, 60001)
        d = dict(kind="extend", n=_log(rng, 11, 230), mean=m, sd=m // 4, lo=m // 3, hi=100000,
                 err=round(rng.uniform(0.03, 0.05), 4), ins=2, dele=2, erate=0.12)
    elif kind == "kmers":
        g = _log(rng, 50_000, 4_000_000)
        c = round(rng.uniform(10, 30), 1)
        d = dict(kind="kmers", genome=g, coverage=c, mean=rng.randrange(5000, 18001), sd=2000, err=0.005,
                 copies=g // 250_000, tandem=0.02, min_count=int(10 * c))
    elif kind == "store":
        d = dict(kind="store", n=_log(rng, 1000, 1_500_000), reads=_log(rng, 100, 300_000), erate=rng.choice([0.045, 1.0]))
    else:
        d = dict(kind="train", n=_log(rng, 1000, 60_000), pos=round(rng.uniform(0.05, 0.3), 3))
    d.pop("name", None)
    return d


# ------------------------------------------------------------------------- read sets
def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed & 0x7FFFFFFF)
    return g


def _rand(g, n):
    return torch.rand(n, generator=g, device=DEVICE)


def _below(g, n, size):
    return torch.randint(0, max(int(n), 1), (int(size),), generator=g, device=DEVICE)


def _genome(g, n, copies=0, tandem=0.0):
    """n base codes: iid, `copies` copies of a 6 kb repeat (1 % divergence, both strands),
    and arrays of a 171-base unit (2 % divergence) over `tandem` of the genome."""
    x = _below(g, 4, n).to(torch.uint8)

    def mutated(y, div):
        hit = _rand(g, y.numel()) < div
        return torch.where(hit, (y + 1 + _below(g, 3, y.numel()).to(torch.uint8)) & 3, y)

    if copies:
        cons = _below(g, 4, 6000).to(torch.uint8)
        slot = n // copies
        at = _below(g, slot - 6000, copies).tolist()
        flip = (_rand(g, copies) < 0.5).tolist()
        for c in range(copies):
            y = mutated(cons, 0.01)
            x[c * slot + at[c]:c * slot + at[c] + 6000] = 3 - y.flip(0) if flip[c] else y
    if tandem:
        unit = _below(g, 4, 171).to(torch.uint8)
        want = int(tandem * n)
        arrays = max(1, want // 20000)
        length = want // arrays
        at = _below(g, n - length, arrays).tolist()
        for c in range(arrays):
            x[at[c]:at[c] + length] = mutated(unit.repeat(length // 171 + 1)[:length], 0.02)
    return x


def _read_count(case):
    return max(2, int(case["genome"] * case["coverage"] / (case["mean"] or 1300)))


def _lengths(g, case, genome):
    """Read lengths by the case's law; their number is that of genome x coverage bases of
    mean-length reads, whatever the seed."""
    lo, hi, mean, sd = float(case["lo"]), float(min(case["hi"], genome)), float(case["mean"]), float(case["sd"])
    law = case["law"]
    n = _read_count(case)
    if law == "lognormal":
        s2 = math.log(1.0 + (sd * sd) / (mean * mean))
        v = torch.exp(math.log(mean) - s2 / 2 + math.sqrt(s2) * torch.randn(n, generator=g, device=DEVICE))
    elif law == "normal":
        v = mean + sd * torch.randn(n, generator=g, device=DEVICE)
    else:
        v = lo / torch.clamp(_rand(g, n), min=1e-9) ** (1 / 1.5)
    return torch.clamp(v, lo, hi).floor().long()


def _sample(g, genome, start, length, err, ins, dele, n_rate=0.0):
    """Reads of genome[start, start + length) with errors, in genome orientation: (codes,
    read offsets [r + 1], source offsets [r + 1], per source base: its output position in
    the read and whether the K bases from it on are free of errors).  Code 4 is N."""
    r = length.numel()
    soff = torch.zeros(r + 1, dtype=torch.long, device=DEVICE)
    soff[1:] = torch.cumsum(length, 0)
    total = int(soff[-1])
    rid = torch.repeat_interleave(torch.arange(r, device=DEVICE), length)
    base = genome[torch.arange(total, device=DEVICE) - (soff[:-1] - start)[rid]]
    u = _rand(g, total)
    s, tot = 1.0, 1.0 + ins + dele
    sub = u < err * s / tot
    isin = (u >= err * s / tot) & (u < err * (s + ins) / tot)
    isdel = (u >= err * (s + ins) / tot) & (u < err)
    base = torch.where(sub, (base + 1 + _below(g, 3, total).to(torch.uint8)) & 3, base)
    count = 1 + isin.long() - isdel.long()
    at = torch.cumsum(count, 0) - count                       # output position of each source base
    out = torch.repeat_interleave(base, count)
    extra = at[isin] + 1
    out[extra] = _below(g, 4, extra.numel()).to(torch.uint8)
    ooff = torch.zeros(r + 1, dtype=torch.long, device=DEVICE)
    ooff[1:] = torch.cumsum(torch.zeros(r, dtype=torch.long, device=DEVICE).index_add_(0, rid, count), 0)
    if n_rate:
        out = torch.where(_rand(g, out.numel()) < n_rate, torch.full_like(out, 4), out)
    bad = torch.cumsum((sub | isin | isdel).long(), 0)
    last = torch.clamp(torch.arange(total, device=DEVICE) + K - 1, max=total - 1)
    clean = (bad[last] - bad + (sub | isin | isdel).long()) == 0
    return out, ooff, soff, at - ooff[:-1][rid], clean


def _host_reads(out, ooff, flip):
    """Base codes in genome orientation -> the host arrays of Overlapper.set_reads: ASCII
    bases in pinned memory, the reads of `flip` reverse-complemented."""
    r = ooff.numel() - 1
    length = ooff[1:] - ooff[:-1]
    rid = torch.repeat_interleave(torch.arange(r, device=DEVICE), length)
    pos = torch.arange(out.numel(), device=DEVICE)
    f = flip[rid]
    src = torch.where(f, ooff[:-1][rid] + ooff[1:][rid] - 1 - pos, pos)
    code = out[src]
    code = torch.where(f & (code < 4), 3 - code, code)
    lut = torch.tensor(list(b"ACGTN"), dtype=torch.uint8, device=DEVICE)
    ascii_ = lut[code.long()]
    host = torch.empty(ascii_.numel(), dtype=torch.uint8, pin_memory=DEVICE == "cuda")
    host.copy_(ascii_)
    return (np.ones(r, np.uint32), length.cpu().numpy().astype(np.uint32), ooff[:-1].cpu().numpy().astype(np.uint64),
            host.numpy())


def _reads(g, case):
    """(genome codes, host read arrays) of a read set."""
    n = int(case["genome"])
    genome = _genome(g, n, case.get("copies", 0), case.get("tandem", 0.0))
    length = _lengths(g, {"law": "normal", "lo": 1000, "hi": 30000, **case}, n)
    start = (_rand(g, length.numel()).double() * (n - length + 1)).long()
    out, ooff, _, _, _ = _sample(g, genome, start, length, case["err"], case.get("ins", 1), case.get("dele", 1),
                                 case.get("n_rate", 0.0))
    flip = _rand(g, length.numel()) < 0.5
    return genome, _host_reads(out, ooff, flip)


def _skip_list(genome, min_count):
    """The canonical K-mers seen min_count times or more in the genome, concatenated."""
    x = genome.long()
    m = x.numel() - K + 1
    fw = torch.zeros(m, dtype=torch.long, device=DEVICE)
    rc = torch.zeros(m, dtype=torch.long, device=DEVICE)
    for j in range(K):
        fw |= x[j:j + m] << (2 * (K - 1 - j))
        rc |= (3 - x[j:j + m]) << (2 * j)
    key, count = torch.unique(torch.minimum(fw, rc), return_counts=True)
    key = key[count >= min_count]
    shift = 2 * torch.arange(K - 1, -1, -1, device=DEVICE)
    lut = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=DEVICE)
    return lut[(key[:, None] >> shift) & 3].cpu().numpy().tobytes()


# ------------------------------------------------------------------------- cases
def prepare(case, seed):
    g = _gen(seed)
    s = {"job": _prepare_job, "extend": _prepare_extend, "kmers": _prepare_kmers, "store": _prepare_store,
         "train": _prepare_train}[case["kind"]](case, g)
    s["kind"] = case["kind"]
    torch.cuda.empty_cache()   # the library allocates beside torch's pool
    return s


def _prepare_job(case, g):
    genome, reads = _reads(g, case)
    refs = int(case["refs"])
    n = len(reads[1])
    p = oic.default_params(kmerLen=K, hashBits=case["bits"], maxHashLoad=case["load"], maxErate=case["erate"],
                           minOlapLen=case["minlen"], maxHashDataLen=case["data"], numThreads=8,
                           partial=case["partial"], uniqueOlapPerPair=1 - case["multi"])
    if refs:
        p.bgnRefID = n // 3
        p.endRefID = min(n, n // 3 + refs)
    ov = oic.Overlapper(p)
    if case["skip"]:
        ov.set_skip_kmers(_skip_list(genome, 11))
    if case["filter"]:
        prm, drop, full, meta = filter_train.load(FILTER)
        ov.set_filter(prm, drop, full, meta["budget"], domain=meta["domain"])
    return dict(ov=ov, reads=reads, n=n, out=np.zeros((int(3 * n * case["coverage"]) + 400_000, 6), np.uint32), used=0)


def _prepare_extend(case, g):
    """n pairs of reads over a common stretch of a random template and, for each pair, an
    exact 22-base match that the two share; S lies on either strand, T on the forward."""
    n = int(case["n"])
    lt = torch.clamp(case["mean"] + case["sd"] * torch.randn(n, generator=g, device=DEVICE), case["lo"], case["hi"]).long()
    ls = torch.clamp(case["mean"] + case["sd"] * torch.randn(n, generator=g, device=DEVICE), case["lo"], case["hi"]).long()
    size = 4_000_000
    genome = _genome(g, size)
    # S starts where it shares at least a third of the shorter read with T.
    share = torch.minimum(ls, lt) // 3
    span = ls + lt - 2 * share
    rel = -ls + share + (_rand(g, n).double() * span).long()        # S start - T start
    t0 = 100_000 + (_rand(g, n).double() * (size - 400_000)).long()
    start = torch.stack([t0 + rel, t0], 1).reshape(-1)              # reads 2i (S) and 2i + 1 (T)
    length = torch.stack([ls, lt], 1).reshape(-1)
    out, ooff, soff, at, clean = _sample(g, genome, start, length, case["err"], case["ins"], case["dele"])
    flip = torch.zeros(2 * n, dtype=torch.bool, device=DEVICE)
    flip[0::2] = _rand(g, n) < 0.5
    reads = _host_reads(out, ooff, flip)
    # A seed: the first of 256 random places of the common stretch that is error-free in
    # both reads for K bases.
    lo, hi = torch.maximum(start[0::2], t0), torch.minimum(start[0::2] + ls, t0 + lt) - K
    p = lo[:, None] + (torch.rand(n, 256, generator=g, device=DEVICE).double() * (hi - lo)[:, None]).long()
    si, ti = soff[0:-1:2][:, None] + p - start[0::2][:, None], soff[1:-1:2][:, None] + p - t0[:, None]
    pick = (clean[si] & clean[ti]).to(torch.uint8).argmax(1, keepdim=True)
    m_start, m_off = at[si.gather(1, pick)][:, 0], at[ti.gather(1, pick)][:, 0]
    p = oic.default_params(kmerLen=K, hashBits=20, maxErate=case["erate"], minOlapLen=500)
    ov = oic.Overlapper(p)
    ov.set_reads(*reads)
    i32 = lambda x: x.cpu().numpy().astype(np.int32)  # noqa: E731
    ids = np.arange(n, dtype=np.uint32)
    prob = (2 * ids + 1, flip[0::2].cpu().numpy().astype(np.uint32), 2 * ids + 2, i32(m_start), i32(m_off),
            np.full(n, K, np.int32))
    return dict(ov=ov, prob=prob)


def _prepare_kmers(case, g):
    _, reads = _reads(g, case)
    ov = oic.Overlapper(oic.default_params(kmerLen=K, hashBits=22))
    ov.set_reads(*reads)
    room = 20_000 + 4000 * case["copies"]
    return dict(ov=ov, n=len(reads[1]), min_count=int(case["min_count"]), out=np.zeros((room, K + 4), np.uint8), used=0)


def _prepare_store(case, g):
    """Records as jobs emit them: a and b near each other in ID order half of the time,
    some pairs with two records, hangs, evalues up to 6 %, both orientations."""
    n, reads = int(case["n"]), int(case["reads"])
    a = 1 + _below(g, reads, n)
    near = 1 + (a - 1 + 1 + _below(g, min(64, reads - 1), n)) % reads
    far = 1 + (a - 1 + 1 + _below(g, reads - 1, n)) % reads
    b = torch.where(_rand(g, n) < 0.5, near, far)
    twin = _rand(g, n) < 0.03
    twin[0] = False
    a, b = torch.where(twin, a.roll(1), a), torch.where(twin, b.roll(1), b)
    hang = lambda: torch.where(_rand(g, n) < 0.5, _below(g, 15000, n), torch.zeros_like(a))  # noqa: E731
    d0 = hang() | (hang() << 21) | (_below(g, 6000, n) << 42) | (_below(g, 2, n) << 58) | (torch.ones_like(a) << 61)
    d1 = hang() | (hang() << 21) | ((1000 + _below(g, 14000, n)) << 42)
    w = torch.stack([a, b, d0 >> 32, d0 & 0xFFFFFFFF, d1 >> 32, d1 & 0xFFFFFFFF], 1)
    return dict(rec=w.cpu().numpy().astype(np.uint32), reads=reads, erate=float(case["erate"]),
                out=np.zeros((2 * n, 6), np.uint32), used=0)


def _prepare_train(case, g):
    """A step in mid-training: the shipped network, features of the filter's ranges (seed
    densities mostly zero, log lengths, log seeds), labels and cost weights, Adam state."""
    n = int(case["n"])
    prm = torch.from_numpy(filter_train.load(FILTER)[0].astype(np.float16)).to(DEVICE)
    x = torch.zeros(n, oic.FILTER_IN, device=DEVICE)
    y = (_rand(g, n) < case["pos"]).float()
    dens = 0.3 * torch.rand(n, 64, generator=g, device=DEVICE)
    x[:, :64] = torch.where(torch.rand(n, 64, generator=g, device=DEVICE) < 0.04, dens, torch.zeros_like(dens))
    x[torch.arange(n, device=DEVICE), _below(g, 64, n)] += 0.75 * y
    x[:, 64:66] = 0.8 + 0.1 * torch.randn(n, 2, generator=g, device=DEVICE)
    x[:, 66] = 0.3 + 0.3 * y + 0.15 * torch.randn(n, generator=g, device=DEVICE)
    wt = torch.where(y > 0, torch.full_like(y, 4.0), 0.05 + torch.clamp(-torch.log(_rand(g, n) + 1e-9), max=20.0))
    f16 = lambda *s: torch.empty(*s, dtype=torch.float16, device=DEVICE)  # noqa: E731
    npar = prm.numel()
    return dict(n=n, x=x.half(), y=y, w=wt, prm=prm, master=prm.float(),
                m=1e-4 * torch.randn(npar, generator=g, device=DEVICE), v=1e-6 * (0.1 + _rand(g, npar)),
                grad=torch.zeros(npar, device=DEVICE), loss=torch.zeros(1, device=DEVICE), h1=f16(n, 128), h2=f16(n, 128),
                g1=f16(n, 128), g2=f16(n, 128), logit=torch.empty(n, device=DEVICE), step=100)


_STATS = ("kmerHitsWithoutOlap", "kmerHitsWithOlap", "kmerHitsSkipped", "multiOverlap", "totalOverlaps",
          "containedOverlaps", "dovetailOverlaps", "seeds", "candidatePairs", "nHashBlocks")
_ADAM = dict(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, decay=1e-5)


def _keep(s, rows):
    """The rows in the caller's own array (its size does not depend on the reads), zeros
    behind them."""
    n, out = len(rows), s["out"]
    out[:n] = rows
    out[n:s["used"]] = 0
    s["used"] = n
    return out


def run(s):
    if s["kind"] == "job":
        ov = s["ov"]
        ov.clear()
        ov.set_reads(*s["reads"])
        ov.run()
        rec, first, counts = oic.store_sort(ov.overlaps(), s["n"])
        st = ov.stats()
        return dict(records=_keep(s, rec).view(np.int32), first=first.view(np.int64), counts=counts,
                    stats={k: int(st[k]) for k in _STATS})
    if s["kind"] == "extend":
        out, kind, delta = s["ov"].extend_batch(*s["prob"])
        return dict(out=out, kind=kind, delta=delta)
    if s["kind"] == "kmers":
        kmers, counts = s["ov"].count_kmers(1, s["n"], s["min_count"])
        rows = np.empty((len(kmers), K + 4), np.uint8)
        rows[:, :K] = np.frombuffer("".join(kmers).encode(), np.uint8).reshape(-1, K)
        rows[:, K:] = counts.view(np.uint8).reshape(-1, 4)
        return dict(kmers=_keep(s, rows))
    if s["kind"] == "store":
        rec, first, counts = oic.store_sort(s["rec"], s["reads"], s["erate"])
        return dict(records=_keep(s, rec).view(np.int32), first=first.view(np.int64), counts=counts)
    p = {k: s[k].data_ptr() for k in ("x", "y", "w", "prm", "master", "m", "v", "grad", "loss", "h1", "h2", "g1", "g2",
                                      "logit")}
    n, st = s["n"], torch.cuda.current_stream().cuda_stream
    s["loss"].zero_()
    oic.mlp_forward(p["prm"], p["x"], n, p["logit"], p["h1"], p["h2"], stream=st)
    oic.mlp_backward(p["prm"], p["x"], p["h1"], p["h2"], p["logit"], p["y"], p["w"], n, p["grad"], p["g1"], p["g2"],
                     p["loss"], stream=st)
    s["step"] += 1
    oic.mlp_adam(p["master"], p["m"], p["v"], p["grad"], p["prm"], _ADAM["lr"], _ADAM["beta1"], _ADAM["beta2"],
                 _ADAM["eps"], 1.0 / n, _ADAM["decay"], s["step"], stream=st)
    return {k: s[k] for k in ("logit", "loss", "h1", "h2", "m", "v", "master", "prm")}


def work(case):
    kind = case["kind"]
    if kind == "job":        # every base read once; each overlap's record read and, with its copy, written
        bases = case["genome"] * case["coverage"]
        mean = case["mean"] or 1500
        share = min(1.0, case["refs"] * mean / bases) if case["refs"] else 1.0
        return {"bytes": bases + share * 72 * (bases / mean) * case["coverage"], "flops": 0}
    if kind == "extend":     # both reads at 2 bits per base, the problem and its result
        return {"bytes": case["n"] * (2 * case["mean"] / 4 + 52), "flops": 0}
    if kind == "kmers":      # both strands at 2 bits per base
        return {"bytes": case["genome"] * case["coverage"] / 2, "flops": 0}
    if kind == "store":      # each record read, it and its copy written
        return {"bytes": 72 * case["n"] + 8 * case["reads"], "flops": 0}
    n, mac = case["n"], 80 * 128 + 128 * 128 + 128
    return {"bytes": n * (160 + 12 + 512) + 30 * oic.FILTER_NPARAM, "flops": 2 * n * (2 * mac + 128 * 128)}


def exact(case, seed):
    """The training step in 64 bits; the other kinds return whole numbers."""
    if case["kind"] != "train":
        return None
    s = _prepare_train(case, _gen(seed))
    q = s["prm"].double()
    part = {k: q[o:o + int(np.prod(shape))].reshape(shape) for k, (o, shape) in oic.FILTER_OFFSETS.items()}
    x, y, wt, n = s["x"].double(), s["y"].double(), s["w"].double(), s["n"]
    h1 = torch.relu(x @ part["w1"].T + part["b1"])
    h2 = torch.relu(h1 @ part["w2"].T + part["b2"])
    z = h2 @ part["w3"] + part["b3"]
    loss = (wt * (torch.clamp(z, min=0) - z * y + torch.log1p(torch.exp(-z.abs())))).sum().reshape(1)
    d = wt * (torch.sigmoid(z) - y)
    z2 = d[:, None] * part["w3"] * (h2 > 0)
    z1 = (z2 @ part["w2"]) * (h1 > 0)
    grad = torch.cat([t.reshape(-1) for t in (z1.T @ x, z1.sum(0), z2.T @ h1, z2.sum(0), d @ h2, d.sum())]) / n
    b1, b2, step = _ADAM["beta1"], _ADAM["beta2"], s["step"] + 1
    m = b1 * s["m"].double() + (1 - b1) * grad
    v = b2 * s["v"].double() + (1 - b2) * grad * grad
    w0 = s["master"].double()
    w = w0 - _ADAM["lr"] * ((m / (1 - b1 ** step)) / (torch.sqrt(v / (1 - b2 ** step)) + _ADAM["eps"]) + _ADAM["decay"] * w0)
    return dict(logit=z, loss=loss, h1=h1, h2=h2, m=m, v=v, master=w, prm=w)
