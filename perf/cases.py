"""Performance cases: what a user of the counter runs, over the range of it.

A case is one use of the public entry points (the `Counter` methods of
kmertreecounter_b200 and its `sizing` module) on seeded synthetic reads of a
stated shape:

  count    FASTQ in device memory -> counts (`Counter.count_device`), then the
           merged count histogram (`Counter.histogram`), which is what the
           counts are mostly made for and what `histogram_tool precise` prints
  sorted   the same with root records sorted by key (`sort_output`)
  learned  the same sized by the learned model beside the count
           (`sizing.BesideSizing`)
  host     the same from pinned host memory (`Counter.count_host`)
  shard    one rank's part of a sharded count: route its reads, then count the
           routed keys it owns (`route_device`, `count_keys_device`)
  sets     many independent read sets of one device buffer in one pass
           (`Counter.count_sets`)
  train    steps of the sizing network's training (`sizing.MLP.train_step`),
           then its weights

The counting outputs are whole numbers that do not depend on the order in
which keys arrive: k-mers read, distinct keys, the histogram of exact counts.
(Which of the two output files a key's first occurrence lies in does depend
on it, so records are compared through the histogram.)
"""
import math

import numpy as np
import torch

import kmertreecounter_b200 as kc
from kmertreecounter_b200 import sizing

HIST_MAX = 10000  # histogram_tool's default range is 1..10000
DIMS = (sizing.N_IN, sizing.N_HID, sizing.N_HID, sizing.N_OUT)
LR, UNDER = 1e-3, 4.0  # the training program's defaults


def _reads(name, kind, k, reads, lo, hi, coverage, gc=0.45, repeats=0.2, error=0.01, buckets=256):
    return {"name": name, "kind": kind, "k": k, "reads": reads, "read_lo": lo, "read_hi": hi, "coverage": coverage,
            "gc": gc, "repeats": repeats, "error": error, "buckets": buckets}


def listed():
    return [
        # the smallest calls: an amplicon or a plasmid, one of many; launches and synchronisations are the cost
        _reads("tiny_k31", "count", 31, 1000, 150, 150, 30.0, repeats=0.0),
        # the plain small shape: 100,000 reads of a 5 Mbp genome
        _reads("small_k31", "count", 31, 100_000, 150, 150, 3.0, gc=0.5, repeats=0.0, error=0.005),
        # trimmed reads of uneven length, the short k of genome profiling
        _reads("ragged_k21", "count", 21, 500_000, 50, 300, 40.0),
        # the genome-scale shape (45% GC, 20% repeats, 30x of 150 bp) at half its size
        _reads("genome_k31", "count", 31, 10_000_000, 150, 150, 30.0),
        # the long-key shape (40% GC, 30% repeats, 50x, 128-bit keys, 4096 buckets) at a tenth
        _reads("long_k63", "count", 63, 6_000_000, 150, 150, 50.0, gc=0.4, repeats=0.3, buckets=4096),
        # 256-bit keys need reads longer than the usual 150
        _reads("wide_k101", "count", 101, 1_000_000, 250, 250, 40.0),
        # sorted root files, for callers that merge or binary-search them
        _reads("sorted_k31", "sorted", 31, 2_000_000, 150, 150, 30.0),
        # structure sizes predicted from the first 1% of the reads, beside the count
        _reads("learned_k31", "learned", 31, 2_000_000, 150, 150, 30.0),
        # a file already read into pinned memory
        _reads("host_k31", "host", 31, 1_500_000, 150, 150, 30.0),
        # one rank of a sharded count
        _reads("shard_k31", "shard", 31, 2_000_000, 150, 150, 30.0),
        # uneven samples counted together: half at k = 21, half at k = 31
        {"name": "sets_48", "kind": "sets", "sets": 48, "reads_lo": 10_000, "reads_hi": 300_000},
        # the sizing network's training: batches of 32 feature rows
        {"name": "train_32", "kind": "train", "steps": 32, "batch": 32},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count"] * 6 + ["sorted", "learned", "host", "shard", "sets", "train"])
    if kind == "sets":
        n = _between(rng, 4, 96)
        lo = _between(rng, 2000, 20_000)
        return {"kind": kind, "sets": n, "reads_lo": lo, "reads_hi": min(400_000, lo * rng.randint(2, 40))}
    if kind == "train":
        return {"kind": kind, "steps": _between(rng, 4, 56), "batch": rng.randint(1, 64)}
    k = rng.choice([21, 25, 27, 31, 31, 32]) if kind != "count" else rng.choice(
        [rng.randint(15, 32), 21, 31, 31, rng.randint(33, 64), 63, rng.randint(65, 95), rng.randint(97, 128)])
    lo = rng.randint(max(50, k + 5), 250)
    hi = lo if rng.random() < 0.5 else rng.randint(lo, 300)
    # bases of a drawn case: up to a third of the largest listed one, less where a key takes more words
    most = {1: 5e8, 2: 3e8, 4: 1.2e8}[1 if k <= 32 else 2 if k <= 64 else 4]
    most = most if kind == "count" else min(most, 3e8)
    reads = _between(rng, 800, most / ((lo + hi) / 2))
    c = _reads(None, kind, k, reads, lo, hi, round(math.exp(rng.uniform(math.log(3), math.log(60))), 2),
               round(rng.uniform(0.3, 0.7), 3), round(rng.choice([0.0, rng.uniform(0.0, 0.4)]), 3),
               round(rng.uniform(0.002, 0.02), 4), rng.choice([256, 256, 4096]))
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs

def _genome(gen, n, gc, repeats):
    """Base codes (A C G T = 0..3) of a random genome, `repeats` of it copies of 1-10 kb templates (1% diverged)."""
    u = torch.rand(n, device="cuda", generator=gen)
    at = (1.0 - gc) / 2
    g = (u >= at).to(torch.uint8) + (u >= 0.5).to(torch.uint8) + (u >= 1.0 - at).to(torch.uint8)
    done, want, top = 0, int(n * repeats), max(50, min(10_000, n // 20))
    r = np.random.default_rng(int(torch.randint(1 << 30, (1,), device="cuda", generator=gen)))
    while done < want:
        length, copies = int(r.integers(max(40, top // 10), top + 1)), int(r.integers(2, 51))
        places = r.permutation(n // length)[:min(copies, (want - done) // length + 1)]  # copies do not overlap
        copies, src = len(places), int(r.integers(0, n - length + 1))
        t = g[src:src + length].clone()
        idx = torch.from_numpy(places * length).cuda()[:, None] + torch.arange(length, device="cuda")
        mut = torch.rand(copies, length, device="cuda", generator=gen) < 0.01
        alt = torch.randint(1, 4, (copies, length), device="cuda", generator=gen, dtype=torch.uint8)
        g[idx] = torch.where(mut, (t + alt) & 3, t.expand(copies, length))
        done += copies * length
    return g


def _fastq(gen, genome, reads, lo, hi, error, n_rate=0.001):
    """FASTQ bytes of `reads` reads at uniform places on either strand: substitutions rising linearly to the 3' end
    (mean `error`), N at n_rate, qualities uniform in 20..40, headers '@r<index>'."""
    letters = torch.tensor(list(b"ACGTN"), dtype=torch.uint8, device="cuda")
    n, parts, first = genome.numel(), [], 0
    col = torch.arange(hi, device="cuda")
    rise = 2.0 * error * (col + 0.5) / hi
    per = max(1, (48 << 20) // (2 * hi + 16))
    while first < reads:
        digits = len(str(first))
        m = min(per, reads - first, 10 ** digits - first)  # one header width per part
        length = torch.randint(lo, hi + 1, (m, 1), device="cuda", generator=gen)
        pos = torch.randint(max(1, n - hi + 1), (m, 1), device="cuda", generator=gen)
        back = torch.rand(m, 1, device="cuda", generator=gen) < 0.5
        code = genome[torch.where(back, pos + length - 1 - col, pos + col).clamp_(0, n - 1)]
        code = torch.where(back, 3 - code, code)
        u = torch.rand(m, hi, device="cuda", generator=gen)
        alt = torch.randint(1, 4, (m, hi), device="cuda", generator=gen, dtype=torch.uint8)
        code = torch.where(u < rise, (code + alt) & 3, code)
        code = torch.where(u > 1.0 - n_rate, 4, code)
        row = torch.empty(m, digits + 2 * hi + 7, dtype=torch.uint8, device="cuda")
        index = torch.arange(first, first + m, device="cuda")
        row[:, 0], row[:, 1], row[:, 2 + digits] = ord("@"), ord("r"), 10
        for d in range(digits):
            row[:, 2 + d] = ((index // 10 ** (digits - 1 - d)) % 10 + 48).to(torch.uint8)
        s, q = 3 + digits, 6 + digits + hi
        row[:, s:s + hi] = letters[code.int()]
        row[:, s + hi:q] = torch.tensor([10, ord("+"), 10], dtype=torch.uint8, device="cuda")
        row[:, q:q + hi] = torch.randint(53, 74, (m, hi), device="cuda", generator=gen, dtype=torch.uint8)
        row[:, q + hi] = 10
        if lo == hi:
            parts.append(row.reshape(-1))
        else:
            keep = torch.ones(row.shape, dtype=torch.bool, device="cuda")
            keep[:, s:s + hi] = col < length
            keep[:, q:q + hi] = col < length
            parts.append(row[keep])
        first += m
    return torch.cat(parts)


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 1_000_003 + 17)
    return gen


def _input(case, seed):
    gen = _generator(seed)
    bases = case["reads"] * (case["read_lo"] + case["read_hi"]) / 2
    genome = _genome(gen, max(2000, int(bases / case["coverage"])), case["gc"], case["repeats"])
    return _fastq(gen, genome, case["reads"], case["read_lo"], case["read_hi"], case["error"])


def _sets_input(case, seed):
    gen, r = _generator(seed), np.random.default_rng(seed)
    parts, sets, lens, off = [], [], [], 0
    for i in range(case["sets"]):
        reads = int(round(math.exp(r.uniform(math.log(case["reads_lo"]), math.log(case["reads_hi"])))))
        length = int(r.integers(50, 301))
        genome = _genome(gen, int(r.integers(1_000_000, 5_000_001)), float(r.uniform(0.3, 0.7)), 0.0)
        f = _fastq(gen, genome, reads, length, length, float(r.uniform(0.005, 0.02)))
        sets.append((off, f.numel(), 21 if i % 2 else 31))
        lens.append(length)
        pad = -f.numel() % 16
        parts += [f, torch.full((pad,), 10, dtype=torch.uint8, device="cuda")]
        off += f.numel() + pad
    return torch.cat(parts), sets


def _train_input(case, seed):
    """Initial weights (the network's own initialisation rule), feature rows and targets of synthetic read sets."""
    r = np.random.default_rng(seed)
    layers = []
    for l in range(3):
        sd = math.sqrt(2.0 / DIMS[l]) * (0.1 if l == 2 else 1.0)
        w = r.standard_normal((DIMS[l], DIMS[l + 1]), np.float32) * np.float32(sd)
        layers.append((w, np.zeros(DIMS[l + 1], np.float32)))
    n = case["steps"] * case["batch"]
    skew = np.exp(r.normal(0.0, 0.7, (8, sizing.MODEL_BUCKETS)))
    pk = 10.0 ** r.uniform(4.5, 6.5, n)
    km = skew[r.integers(0, 8, n)]
    km = r.poisson(np.minimum(km / km.sum(axis=1, keepdims=True) * pk[:, None], 1e6))
    dist = r.uniform(0.1, 0.95, n)
    tab = dist * r.uniform(0.05, 0.5, n)
    kp = km.sum(axis=1)
    fastq = pk * r.uniform(200, 260, n)
    x = sizing.features_batch(km, dist * kp, tab * kp, r.choice([21, 31, 63], n), np.full(n, 150.0), fastq, fastq / 100)
    y = np.empty((n, sizing.N_OUT), np.float32)
    noise = r.normal(0.0, 0.02, (n, sizing.N_OUT)).astype(np.float32)
    y[:, :sizing.MODEL_BUCKETS] = (np.log(dist + 1e-4) / 10.0 + 1.0)[:, None]
    y[:, sizing.MODEL_BUCKETS:] = (np.log(tab + 1e-4) / 10.0 + 1.0)[:, None]
    return layers, x, y + noise


# ------------------------------------------------------------------ the cases

def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        layers, x, y = _train_input(case, seed)
        m = sizing.MLP(max_batch=case["batch"], seed=7)
        m.set_under_weight(UNDER)
        for l, (w, b) in enumerate(layers):
            m.set_layer(l, w, b)
        return {"kind": kind, "model": m, "x": x, "y": y, "steps": case["steps"], "batch": case["batch"]}
    if kind == "sets":
        data, sets = _sets_input(case, seed)
        s = {"kind": kind, "data": data, "sets": sets, "counter": kc.Counter(k=31)}
    else:
        data = _input(case, seed)
        s = {"kind": kind, "data": data, "counter": kc.Counter(
            k=case["k"], n_buckets=case["buckets"], sort_output=int(kind == "sorted"),
            sizing=kc.KC_SIZING_LEARNED if kind == "learned" else kc.KC_SIZING_SAMPLED)}
        if kind == "host":
            s["data"] = torch.empty(data.numel(), dtype=torch.uint8, pin_memory=True).copy_(data)
        if kind == "learned":
            s["beside"] = sizing.BesideSizing(s["counter"], sizing.MLP.load(), case["k"], case["read_hi"])
            s["beside"].target = (data.data_ptr(), data.numel())
    torch.cuda.synchronize()  # the counter works on a stream of its own
    torch.cuda.empty_cache()  # the counter allocates beside torch
    return s


def _spectrum(c):
    hist, distinct = c.histogram(1, HIST_MAX)
    return {"kmers": int(c.stats.total_kmers), "distinct": int(distinct), "hist": hist.astype(np.int64)}


def run(s):
    kind = s["kind"]
    if kind == "train":
        m, b = s["model"], s["batch"]
        losses = [m.train_step(s["x"][i * b:(i + 1) * b], s["y"][i * b:(i + 1) * b], LR) for i in range(s["steps"])]
        layers = [m.get_layer(l) for l in range(3)]
        return {"loss": np.array(losses, np.float32), "w": [w for w, _ in layers], "b": [b for _, b in layers]}
    c, data = s["counter"], s["data"]
    if kind == "sets":
        return {"kmers": np.array([r.total_kmers for r in c.count_sets(data.data_ptr(), s["sets"])], np.int64)}
    if kind == "host":
        c.count_host_ptr(data.data_ptr(), data.numel())
    elif kind == "shard":
        counts = c.route_device(data.data_ptr(), data.numel())
        addr, n = c.routed_keys()
        # the exchange's place: this rank's own buffer for the keys it receives
        if s.get("keys") is None or s["keys"].numel() < n:
            s["keys"] = torch.empty(n + n // 8, dtype=torch.int64, device="cuda")
        c.copy_routed(s["keys"].data_ptr(), 8 * n)
        c.count_keys_device(s["keys"].data_ptr(), n, counts)
    else:
        c.count_device(data.data_ptr(), data.numel())
    return _spectrum(c)


def work(case):
    """Counting: the FASTQ read once, the packed first occurrences and root records written once (about a quarter of the
    k-mers are first occurrences and a twentieth root records at the shapes above).  Training: a step reads its batch
    and reads and writes weights, gradient moments and their 16-bit copy."""
    if case["kind"] == "train":
        p = sum(DIMS[l] * DIMS[l + 1] for l in range(3))
        step = 4.0 * case["batch"] * (DIMS[0] + DIMS[3]) + 26.0 * p
        return {"bytes": case["steps"] * step, "flops": 6.0 * p * case["batch"] * case["steps"]}
    if case["kind"] == "sets":
        lo, hi = case["reads_lo"], case["reads_hi"]
        reads = case["sets"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        length, k, rest = 175.0, 26, 7
    else:
        reads, k = case["reads"], case["k"]
        length, rest = (case["read_lo"] + case["read_hi"]) / 2, 6 + len(str(reads))
    kmers = reads * max(0.0, length - k + 1)
    return {"bytes": reads * (2 * length + rest) + kmers * (0.25 * kc.packed_bytes(k) + 0.05 * kc.record_bytes(k)),
            "flops": 0}


def exact(case, seed):
    """Training in 64 bits, plain torch.  Adam divides a gradient by its own size, so a gradient near zero that 16-bit
    activations round the other way moves its weight by a whole step in the other direction: the biases (zero at first)
    and the small last layer are mostly made of such steps and have no value to be held to.  The counting cases return
    whole numbers only."""
    if case["kind"] != "train":
        return None
    layers, x, y = _train_input(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    put = lambda a: torch.from_numpy(a).to(dev, torch.float64)  # noqa: E731
    p = [put(a) for w, b in layers for a in (w, b)]
    m, v = [torch.zeros_like(a) for a in p], [torch.zeros_like(a) for a in p]
    losses, n = [], case["batch"]
    for i in range(case["steps"]):
        xb, yb = put(x[i * n:(i + 1) * n]), put(y[i * n:(i + 1) * n])
        h1 = (xb @ p[0] + p[1]).clamp_min(0)
        h2 = (h1 @ p[2] + p[3]).clamp_min(0)
        e = h2 @ p[4] + p[5] - yb
        w = torch.where(e < 0, UNDER, 1.0)
        losses.append(float((w * e * e).mean()))
        d3 = 2.0 * w * e / e.numel()
        d2 = (d3 @ p[4].T) * (h2 > 0)
        d1 = (d2 @ p[2].T) * (h1 > 0)
        grads = [xb.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ d3, d3.sum(0)]
        c1, c2 = 1.0 - 0.9 ** (i + 1), 1.0 - 0.999 ** (i + 1)
        for a, g, s, t in zip(p, grads, m, v):
            s.mul_(0.9).add_(g, alpha=0.1)
            t.mul_(0.999).addcmul_(g, g, value=0.001)
            a.sub_(LR * (s / c1) / ((t / c2).sqrt() + 1e-8))
    return {"loss": torch.tensor(losses, dtype=torch.float64), "w": [p[0].cpu(), p[2].cpu(), None], "b": [None] * 3}
