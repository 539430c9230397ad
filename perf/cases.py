"""The calls a user of this engine makes, at the sizes it makes them.

A case names an entry point (``call``) and the shape of one synthetic batch:

* ``pair``      ``Engine.pair``: one read against one haplotype, the smallest call
* ``batch``     ``Engine.batch``: regions in host buffers in, log10 likelihoods out
* ``resident``  ``Engine.upload`` once, then ``DeviceBatch.run`` + ``download``
* ``service``   ``Service.submit`` of every region by itself, then ``wait`` for each

The synthetic model is that of ``rodv_b200.workloads``: a region has a locus of
random bases; its haplotypes are mutated copies of it and its reads mutated
substrings of a random haplotype (``sub`` substitutions and ``indel`` 1-3 base
indels per base); base qualities are uniform in [q_lo, q_hi], and the gap
qualities are 45/45/10 on every base (``gaps`` = "flat") or drawn per base as
recalibrated reads and the golden file have them ("per_base").  ``related`` =
False takes the reads from elsewhere, so that most likelihoods underflow FP32.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import rodv_b200
from rodv_b200.batch import REGION_DTYPE, Batch

DEVICE = "cuda"

# One batch shape; a case overrides what it needs.
DEFAULTS = {
    "call": "batch", "regions": 1, "haps_lo": 2, "haps_hi": 16, "reads_lo": 20, "reads_hi": 200,
    "hap_lo": 100, "hap_hi": 600, "len_lo": 50, "len_hi": 250, "sub": 0.01, "indel": 0.001,
    "q_lo": 10, "q_hi": 40, "gaps": "flat", "n_rate": 0.0, "related": True, "use_double": False,
}


def _case(name, **over):
    return {"name": name, **DEFAULTS, **over}


def listed():
    return [
        # one read against one haplotype (compute_likelihoods of a caller that
        # has no batch): latency of the whole call
        _case("pair", call="pair", haps_lo=1, haps_hi=1, reads_lo=1, reads_hi=1, hap_lo=300,
              hap_hi=300, len_lo=151, len_hi=151),
        # one active region at a time, as schedule_pairhmm is called: the
        # benchmark's plain region of 64 reads x 8 haplotypes
        _case("region", haps_lo=8, haps_hi=8, reads_lo=64, reads_hi=64, hap_lo=250, hap_hi=400,
              len_lo=150, len_hi=150),
        # a handful of regions of recalibrated reads (gap qualities per base,
        # some N bases): a caller's small work list
        _case("regions_recal", regions=7, haps_lo=1, haps_hi=9, reads_lo=3, reads_hi=61,
              hap_lo=81, hap_hi=420, len_lo=30, len_hi=251, q_lo=6, q_hi=43, gaps="per_base",
              n_rate=0.002),
        # an ordinary work list: 100 regions of uneven lengths
        _case("regions", regions=100),
        # the benchmark's uneven batch at a quarter of its regions: the
        # pipelined host path
        _case("regions_many", regions=2500),
        # the same shape kept on the device (re-evaluated likelihoods)
        _case("resident", call="resident", regions=500),
        # recalibrated reads at scale: the kernels with per-row gap priors
        _case("recal_many", regions=300, q_lo=6, q_hi=43, gaps="per_base", n_rate=0.0005),
        # short reads (36-101 bases) of older instruments and amplicons
        _case("short_reads", regions=400, reads_lo=10, reads_hi=300, haps_lo=2, haps_hi=12,
              hap_lo=80, hap_hi=250, len_lo=36, len_hi=101),
        # every pair in double precision (schedule_pairhmm's use_double)
        _case("double", regions=50, use_double=True),
        # low-quality reads against unrelated haplotypes: FP32 underflows and
        # the FP64 pass does the work, one pair per region
        _case("underflow", regions=40000, haps_lo=1, haps_hi=1, reads_lo=1, reads_hi=1,
              hap_lo=400, hap_hi=400, len_lo=250, len_hi=250, q_lo=2, q_hi=8, related=False),
        # long reads at 5% differences: multi-pass sweeps, rescued in FP64
        _case("long_pairs", regions=1500, haps_lo=1, haps_hi=1, reads_lo=1, reads_hi=1,
              hap_lo=2000, hap_hi=5000, len_lo=1000, len_hi=2000, sub=0.05, indel=0.01),
        # requests arriving one region at a time at the streaming service
        _case("service", call="service", regions=150, haps_lo=1, haps_hi=32, reads_lo=1,
              reads_hi=300, hap_lo=100, hap_hi=800),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: a listed kind at other sizes, regions and lengths spread
    over the listed range."""
    kind = rng.choice(["pair", "small", "batch", "batch", "recal", "resident", "short", "double",
                       "underflow", "long", "long_clean", "service"])
    c = dict(DEFAULTS)
    if kind == "pair":
        h, n = _log_int(rng, 40, 800), _log_int(rng, 20, 500)
        c.update(call="pair", haps_lo=1, haps_hi=1, reads_lo=1, reads_hi=1, hap_lo=h, hap_hi=h,
                 len_lo=n, len_hi=n, gaps=rng.choice(["flat", "per_base"]),
                 use_double=rng.random() < 0.2)
    elif kind == "small":
        c.update(regions=rng.randint(1, 12), haps_lo=1, haps_hi=rng.randint(1, 20), reads_lo=1,
                 reads_hi=_log_int(rng, 2, 250), hap_lo=rng.randint(60, 200),
                 hap_hi=rng.randint(201, 700), len_lo=rng.randint(20, 120),
                 len_hi=rng.randint(121, 300), gaps=rng.choice(["flat", "flat", "per_base"]))
    elif kind in ("batch", "resident"):
        c.update(call=kind, regions=_log_int(rng, 10, 2000 if kind == "batch" else 700),
                 haps_hi=rng.randint(3, 16), reads_hi=rng.randint(30, 200),
                 hap_lo=rng.randint(60, 250), hap_hi=rng.randint(251, 600),
                 len_lo=rng.randint(30, 130), len_hi=rng.randint(131, 254))
    elif kind == "recal":
        c.update(regions=_log_int(rng, 10, 400), haps_hi=rng.randint(3, 16),
                 reads_hi=rng.randint(30, 200), len_hi=rng.randint(100, 250), q_lo=6, q_hi=43,
                 gaps="per_base", n_rate=rng.choice([0.0, 0.002]))
    elif kind == "short":
        c.update(regions=_log_int(rng, 20, 600), reads_lo=5, reads_hi=rng.randint(20, 300),
                 haps_hi=rng.randint(2, 12), hap_lo=60, hap_hi=rng.randint(100, 300),
                 len_lo=rng.randint(18, 40), len_hi=rng.randint(45, 126))
    elif kind == "double":
        c.update(regions=_log_int(rng, 2, 80), reads_hi=rng.randint(30, 200), use_double=True,
                 gaps=rng.choice(["flat", "flat", "per_base"]))
    elif kind == "underflow":
        n, h = rng.randint(180, 250), rng.randint(200, 500)
        c.update(regions=_log_int(rng, 500, 50000), haps_lo=1, haps_hi=1, reads_lo=1, reads_hi=1,
                 hap_lo=h, hap_hi=h + rng.randint(0, 100), len_lo=n, len_hi=n, q_lo=2, q_hi=8,
                 related=False)
    elif kind in ("long", "long_clean"):
        n, h = rng.randint(300, 1500), rng.randint(2000, 4000)
        c.update(regions=_log_int(rng, 20, 1500), haps_lo=1, haps_hi=1, reads_lo=1, reads_hi=1,
                 hap_lo=h, hap_hi=h + rng.randint(0, 1000), len_lo=n,
                 len_hi=n + rng.randint(0, 500), sub=0.05, indel=0.01)
        if kind == "long_clean":  # accurate long reads: most stay in FP32
            c.update(regions=_log_int(rng, 1, 60), haps_hi=rng.randint(1, 6),
                     reads_hi=rng.randint(1, 12), sub=0.001, indel=0.0002, q_lo=25)
    else:
        c.update(call="service", regions=_log_int(rng, 20, 200), haps_lo=1,
                 haps_hi=rng.randint(2, 32), reads_lo=1, reads_hi=rng.randint(10, 300),
                 hap_hi=rng.randint(200, 800))
    c["kind"] = kind
    return c


# ---------------------------------------------------------------------------
# Inputs: one batch from a seed, generated on the GPU, kept in host buffers.
# ---------------------------------------------------------------------------
def _ranges(start, length):
    """start[k] + [0, length[k]) for every k, concatenated, and each value's k."""
    k = torch.repeat_interleave(torch.arange(len(length), device=DEVICE), length)
    first = torch.cumsum(length, 0) - length
    return start[k] + torch.arange(len(k), device=DEVICE) - first[k], k


def _mutated(gen, seq, start, length, sub, indel):
    """Substrings seq[start[k], +length[k]) with substitutions and 1-3 base
    indels: (codes, lengths)."""
    at, k = _ranges(start, length)
    codes = seq[at]
    n = len(codes)
    rnd = torch.rand(n, generator=gen, device=DEVICE)
    other = torch.randint(1, 4, (n,), generator=gen, device=DEVICE, dtype=torch.uint8)
    codes = torch.where(rnd < sub, (codes + other) % 4, codes)
    if indel <= 0:
        return codes, length
    first = torch.cumsum(length, 0) - length
    copies = torch.ones(n, dtype=torch.int64, device=DEVICE)
    event = torch.rand(n, generator=gen, device=DEVICE)
    size = torch.randint(1, 4, (n,), generator=gen, device=DEVICE)
    copies += torch.where(event < indel / 2, size, torch.zeros_like(size))
    gone = event > 1 - indel / 2
    for d in range(3):
        hit = torch.zeros_like(gone)
        hit[d:] = gone[:n - d] & (size[:n - d] > d)
        copies[hit] = 0
    copies[first] = torch.clamp(copies[first], min=1)
    src = torch.repeat_interleave(torch.arange(n, device=DEVICE), copies)
    run = torch.cumsum(copies, 0) - copies
    added = torch.arange(len(src), device=DEVICE) > run[src]
    extra = torch.randint(0, 4, (len(src),), generator=gen, device=DEVICE, dtype=torch.uint8)
    out = torch.where(added, extra, codes[src])
    return out, torch.zeros_like(length).index_add_(0, k[src], torch.ones_like(src))


def _host(t, dtype=np.uint8):
    return np.ascontiguousarray(t.cpu().numpy().astype(dtype, copy=False))


def _counts(case):
    """Haplotypes and reads of every region: of the case, not of the seed, so
    that every seed's result has one shape."""
    rng = np.random.default_rng(case["regions"])
    return (rng.integers(case["haps_lo"], case["haps_hi"] + 1, size=case["regions"]),
            rng.integers(case["reads_lo"], case["reads_hi"] + 1, size=case["regions"]))


def _make(case, seed):
    """The case's batch of this seed."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)

    def ints(lo, hi, n):
        return torch.randint(lo, hi + 1, (n,), generator=gen, device=DEVICE)

    g = case["regions"]
    locus_len = ints(case["hap_lo"], case["hap_hi"], g)
    locus_off = torch.cumsum(locus_len, 0) - locus_len
    locus = torch.randint(0, 4, (int(locus_len.sum()),), generator=gen, device=DEVICE,
                          dtype=torch.uint8)
    num_haps, num_reads = (torch.from_numpy(x).to(DEVICE) for x in _counts(case))
    hap_region = torch.repeat_interleave(torch.arange(g, device=DEVICE), num_haps)
    read_region = torch.repeat_interleave(torch.arange(g, device=DEVICE), num_reads)
    haps, hap_len = _mutated(gen, locus, locus_off[hap_region], locus_len[hap_region],
                             case["sub"], case["indel"])
    hap_off = torch.cumsum(hap_len, 0) - hap_len
    hap_start = torch.cumsum(num_haps, 0) - num_haps
    n = len(read_region)
    want = ints(case["len_lo"], case["len_hi"], n)
    if case["related"]:
        pick = (torch.rand(n, generator=gen, device=DEVICE) * num_haps[read_region]).long()
        src = hap_start[read_region] + torch.minimum(pick, num_haps[read_region] - 1)
        want = torch.minimum(want, hap_len[src])
        room = hap_len[src] - want + 1
        at = (torch.rand(n, generator=gen, device=DEVICE) * room).long()
        reads, read_len = _mutated(gen, haps, hap_off[src] + torch.minimum(at, room - 1), want,
                                   case["sub"], case["indel"])
    else:
        reads = torch.randint(0, 4, (int(want.sum()),), generator=gen, device=DEVICE,
                              dtype=torch.uint8)
        read_len = want
    read_off = torch.cumsum(read_len, 0) - read_len
    total = len(reads)
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=DEVICE)
    hap_bases, read_bases = letters[haps.long()], letters[reads.long()]
    if case["n_rate"] > 0:
        for s in (hap_bases, read_bases):
            s[torch.rand(len(s), generator=gen, device=DEVICE) < case["n_rate"]] = ord("N")
    quals = _host(ints(case["q_lo"], case["q_hi"], total).to(torch.uint8))
    if case["gaps"] == "flat":
        gaps = [np.full(total, v, np.uint8) for v in (45, 45, 10)]
    else:
        gaps = [_host(ints(lo, hi, total).to(torch.uint8))
                for lo, hi in ((30, 45), (30, 45), (8, 14))]
    regions = np.zeros(g, dtype=REGION_DTYPE)
    read_start = torch.cumsum(num_reads, 0) - num_reads
    for name, v in zip(REGION_DTYPE.names, (hap_start, num_haps, read_start, num_reads)):
        regions[name] = v.cpu().numpy()
    return Batch(regions, _host(hap_bases), _host(hap_off, np.uint64), _host(hap_len, np.uint32),
                 _host(read_bases), quals, *gaps, _host(read_off, np.uint64),
                 _host(read_len, np.uint32))


# ---------------------------------------------------------------------------
# Passes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _service():
    """The program's streaming service (kept while the program runs)."""
    return rodv_b200.Service(device_memory_budget=8 << 30)


def prepare(case, seed):
    b = _make(case, seed)
    state = {"call": case["call"], "use_double": bool(case["use_double"]), "batch": b,
             "engine": rodv_b200.default_engine()}
    if case["call"] == "pair":
        state["pair"] = [b.hap_bases, b.read_bases, b.base_quals, b.ins_quals, b.del_quals,
                         b.gcp_quals]
    elif case["call"] == "resident":
        state["resident"] = state["engine"].upload(b)
    elif case["call"] == "service":
        state["service"] = _service()
        state["requests"] = _split(b)
    return state


def _split(b):
    """Every region as a batch of its own over the same buffers."""
    out = []
    for r in b.regions:
        h0, h1 = int(r["hap_start"]), int(r["hap_start"]) + int(r["num_haps"])
        r0, r1 = int(r["read_start"]), int(r["read_start"]) + int(r["num_reads"])
        region = np.array([(0, h1 - h0, 0, r1 - r0)], dtype=REGION_DTYPE)
        out.append(Batch(region, b.hap_bases, b.hap_offsets[h0:h1], b.hap_lengths[h0:h1],
                         b.read_bases, b.base_quals, b.ins_quals, b.del_quals, b.gcp_quals,
                         b.read_offsets[r0:r1], b.read_lengths[r0:r1]))
    return out


def run(state):
    engine, call = state["engine"], state["call"]
    if call == "pair":
        return engine.pair(*state["pair"], use_double=state["use_double"])
    if call == "resident":
        state["resident"].run()
        return state["resident"].download()
    if call == "service":
        service = state["service"]
        tickets = [service.submit(r) for r in state["requests"]]
        return np.concatenate([service.wait(t) for t in tickets])
    return engine.batch(state["batch"], use_double=state["use_double"])


def _mean(lo, hi):
    return 0.5 * (lo + hi)


def work(case):
    """Of one pass: 12 operations per cell (M 4 mul + 2 add, I 2 + 1, D 2 + 1);
    the bases and four qualities of each read, the haplotype bases and a
    double per pair.  Lengths are the means of what the seeds draw."""
    haps, reads = _counts(case)
    h, r, pairs = int(haps.sum()), int(reads.sum()), int((haps * reads).sum())
    hap, read = _mean(case["hap_lo"], case["hap_hi"]), _mean(case["len_lo"], case["len_hi"])
    if case["related"]:
        read = min(read, hap)
    return {"bytes": 5 * r * read + h * hap + 8 * pairs, "flops": 12.0 * pairs * hap * read}


# ---------------------------------------------------------------------------
# The same likelihoods in 64 bits with plain torch: anti-diagonals of all
# pairs of a chunk at once.
# ---------------------------------------------------------------------------
def _match_to_match():
    """P(no gap opened) by (ins, del) quality: 1 - (10^-ins/10 + 10^-del/10),
    the sum by the model's log10 table of step 1e-4 (differences up to 8)."""
    q = np.arange(128)
    lo, hi = np.minimum.outer(q, q), np.maximum.outer(q, q)
    diff = 0.1 * hi - 0.1 * lo
    steps = np.floor(diff * (1.0 / 1e-4) + 0.5)
    s = -0.1 * lo + np.where(diff >= 8.0, 0.0, np.log10(1.0 + 10.0 ** (-steps * 1e-4)))
    p = np.minimum(1.0, 10.0 ** s)
    with np.errstate(divide="ignore"):
        return 10.0 ** (np.log1p(-p) / np.log(10.0))


def _padded(flat, off, length, width, left, fill):
    """Rows of a [n, left + width] tensor: `left` fill values, then each
    sequence, then fill values."""
    n = len(length)
    out = torch.full((n, left + width), fill, dtype=flat.dtype, device=DEVICE)
    at, k = _ranges(off, length)
    out[k, left + at - off[k]] = flat[at]
    return out


def _exact_chunk(hap, hap_len, read, read_len, q, ins, dele, gcp, mm_table):
    """log10 likelihoods of B pairs: hap [B, H] and read [B, L] letters."""
    b, h_max = hap.shape
    l_max = read.shape[1]
    f = torch.float64
    prob = torch.tensor(10.0 ** (-np.arange(128) / 10.0), dtype=f, device=DEVICE)
    err = prob[q]
    match, mismatch = 1 - err, err / 3
    any_read = read == ord("N")
    match = torch.where(read == 0, torch.zeros_like(match), match)
    mm, gapm = mm_table[ins, dele], 1 - prob[gcp]
    mi, ii, md = prob[ins], prob[gcp], prob[dele]
    # columns left of 1 and right of H carry letter 0: emission 0
    wide = torch.zeros((b, h_max + 2 * l_max), dtype=hap.dtype, device=DEVICE)
    wide[:, l_max:l_max + h_max] = hap
    wide = wide.flip(1)
    init = 2.0 ** 1020 / hap_len.to(f)

    def zeros():
        return torch.zeros((b, l_max + 1), dtype=f, device=DEVICE)

    # state of the last two anti-diagonals, rows 0..L
    m1, i1, d1, m2, i2, d2 = (zeros() for _ in range(6))
    d1[:, 0] = init
    total = torch.zeros(b, dtype=f, device=DEVICE)
    rows = torch.arange(b, device=DEVICE)
    steps = h_max + l_max
    for d in range(1, steps + 1):
        # letters of columns d-1, d-2, ..., d-L (from 1) beside rows 1..L
        off = h_max + l_max + 1 - d
        col = wide[:, off:off + l_max]
        hit = (col == read) | any_read | (col == ord("N"))
        e = torch.where(hit, match, mismatch) * (col != 0)
        m, i, dd = zeros(), zeros(), zeros()
        m[:, 1:] = e * (mm * m2[:, :-1] + gapm * (i2[:, :-1] + d2[:, :-1]))
        i[:, 1:] = mi * m1[:, :-1] + ii * i1[:, :-1]
        dd[:, 1:] = md * m1[:, 1:] + ii * d1[:, 1:]
        dd[:, 0] = init
        m2, i2, d2, m1, i1, d1 = m1, i1, d1, m, i, dd
        j = d - read_len
        last = m[rows, read_len] + i[rows, read_len]
        total += torch.where((j >= 1) & (j <= hap_len), last, torch.zeros_like(last))
    return torch.log10(total) - math.log10(2.0 ** 1020)


def exact(case, seed):
    cells = work(case)["flops"] / 12
    if cells > 3e10:  # over about 20 seconds
        return None
    b = _make(case, seed)
    r = b.regions
    pairs_of = r["num_haps"].astype(np.int64) * r["num_reads"]
    region = np.repeat(np.arange(len(r)), pairs_of)
    k = np.arange(len(region)) - np.repeat(np.cumsum(pairs_of) - pairs_of, pairs_of)
    hap = r["hap_start"][region] + k // r["num_reads"][region]
    read = r["read_start"][region] + k % r["num_reads"][region]
    order = np.lexsort((b.hap_lengths[hap], b.read_lengths[read]))
    out = torch.empty(len(region), dtype=torch.float64, device=DEVICE)

    def dev(a):
        return torch.from_numpy(a.astype(np.int64)).to(DEVICE)

    hap_len, hap_off = dev(b.hap_lengths), dev(b.hap_offsets)
    read_len, read_off = dev(b.read_lengths), dev(b.read_offsets)
    hb = torch.from_numpy(b.hap_bases).to(DEVICE)
    fields = [torch.from_numpy(x).to(DEVICE) for x in (b.read_bases, b.base_quals, b.ins_quals,
                                                       b.del_quals, b.gcp_quals)]
    mm_table = torch.tensor(_match_to_match(), dtype=torch.float64, device=DEVICE)
    at = 0
    while at < len(order):
        # about 12 million rows in a chunk
        n = max(1, int(1.2e7 // max(1, int(b.read_lengths[read[order[min(len(order) - 1, at +
                                                                        40000)]]]))))
        pick = order[at:at + n]
        hs, rs = dev(hap[pick]), dev(read[pick])
        hl, rl = hap_len[hs], read_len[rs]
        w = int(rl.max())
        read_fields = [_padded(x, read_off[rs], rl, w, 0, 0) for x in fields]
        letters, quals = read_fields[0], [x.long() for x in read_fields[1:]]
        out[torch.from_numpy(pick).to(DEVICE)] = _exact_chunk(
            _padded(hb, hap_off[hs], hl, int(hl.max()), 0, 0), hl, letters, rl, *quals, mm_table)
        at += n
    v = out.cpu().numpy()
    return float(v[0]) if case["call"] == "pair" else v
