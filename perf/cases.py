"""The work that a user has this framework do, as cases that can be timed and compared.

A case is one call (or one burst of calls) through the public Python interface: `galn_b200.aln` on a resident
index, a `Server` with requests in flight, `index_text` (the device part of `galn index` with its files), or
`Index.sa2pos` (samse's coordinate step). Genomes and reads are synthetic, with the shapes of the aln workloads
in galn_b200/synth.py, drawn on the GPU because they are made often. A genome depends on its kind and length
alone, since a program keeps its index; the reads, rows or sequences of a case depend on the seed.
"""
from __future__ import annotations

import math
import os
import tempfile
from collections import OrderedDict

import numpy as np
import torch

import galn_b200
from galn_b200 import synth

DEFAULT, ADNA, DIVERGENT = [], synth.ADNA_OPTS, synth.DIVERGENT_OPTS

# Per kind of reads: options, and the occurrence blocks (32 bytes) that one read's search looks up on average, as
# the search counts them. Each lookup counts the four bases before a position of the BWT.
KINDS = {
    "plain": dict(opts=DEFAULT, blocks=730),
    "mixed": dict(opts=DEFAULT, blocks=870),
    "mixed_adna": dict(opts=ADNA, blocks=5_200),
    "adna": dict(opts=ADNA, blocks=2_800),
    "divergent": dict(opts=DIVERGENT, blocks=570_000),
    "genome": dict(opts=DEFAULT, blocks=2_800),
}
# Integer operations of one lookup that no layout avoids: per base an and, a population count and an add, over
# two positions and two words.
OPS_PER_BLOCK = 24


def listed():
    return [
        # an interactive query: a handful of reads against a small genome, where latency is all there is
        dict(name="aln_few", task="aln", genome="uniform", bp=1_000_000, kind="plain", reads=64, length=100, trace=False),
        # a small resequencing run: the plain configuration, 20,000 x 100 bp on 1 Mbp, default options
        dict(name="aln_plain", task="aln", genome="uniform", bp=1_000_000, kind="plain", reads=20_000, length=100,
             trace=False),
        # one bwa batch (0x40000 reads) of ancient DNA, as a reader thread hands it over
        dict(name="aln_adna_batch", task="aln", genome="adna", bp=100_000_000, kind="adna", reads=262_144, length=0,
             trace=False),
        # the whole aDNA configuration in one call
        dict(name="aln_adna_2m", task="aln", genome="adna", bp=100_000_000, kind="adna", reads=2_000_000, length=0,
             trace=False),
        # the high-divergence configuration (-N: every read is searched to the end), a part of its reads
        dict(name="aln_divergent", task="aln", genome="adna", bp=100_000_000, kind="divergent", reads=10_000, length=100,
             trace=False),
        # the genome-scale configuration at a tenth of its genome: an index past L2, repeats, ambiguous bases
        dict(name="aln_genome", task="aln", genome="genome", bp=310_000_000, kind="genome", reads=200_000, length=150,
             trace=False),
        # reads of a request stream (36-150 bp) with the per-read trace hashes on: the library's default, and --verify
        dict(name="aln_mixed_trace", task="aln", genome="adna", bp=100_000_000, kind="mixed", reads=50_001, length=0,
             trace=True),
        # serving: a burst of requests of log-uniform sizes, half default and half aDNA options, on one index
        dict(name="serve_burst", task="serve", genome="adna", bp=100_000_000, requests=12, reads=150_000),
        # `galn index` on a bacterial-size sequence, and on the aDNA configuration's 100 Mbp
        dict(name="index_small", task="index", genome="uniform", bp=1_000_003),
        dict(name="index_100m", task="index", genome="adna", bp=100_000_000),
        # genome positions of hits: a small set, and one row per read of the aDNA configuration
        dict(name="pos_small", task="pos", genome="adna", bp=100_000_000, rows=5_000),
        dict(name="pos_2m", task="pos", genome="adna", bp=100_000_000, rows=2_000_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["plain", "adna", "adna", "divergent", "genome", "mixed", "serve", "index", "pos"])
    if what == "plain":
        return dict(task="aln", genome="uniform", bp=_log_int(rng, 500_000, 10_000_000), kind="plain",
                    reads=_log_int(rng, 16, 200_000), length=rng.randint(36, 150), trace=rng.random() < 0.25)
    if what == "adna":
        return dict(task="aln", genome="adna", bp=_log_int(rng, 5_000_000, 100_000_000), kind="adna",
                    reads=_log_int(rng, 500, 1_500_000), length=0, trace=rng.random() < 0.25)
    if what == "divergent":
        return dict(task="aln", genome="adna", bp=_log_int(rng, 5_000_000, 100_000_000), kind="divergent",
                    reads=_log_int(rng, 200, 10_000), length=rng.randint(70, 100), trace=False)
    if what == "genome":
        return dict(task="aln", genome="genome", bp=_log_int(rng, 20_000_000, 310_000_000), kind="genome",
                    reads=_log_int(rng, 2_000, 200_000), length=rng.randint(100, 150), trace=False)
    if what == "mixed":
        return dict(task="aln", genome="adna", bp=_log_int(rng, 5_000_000, 100_000_000),
                    kind=rng.choice(["mixed", "mixed_adna"]), reads=_log_int(rng, 500, 100_000), length=0,
                    trace=rng.random() < 0.5)
    if what == "serve":
        return dict(task="serve", genome="adna", bp=_log_int(rng, 5_000_000, 100_000_000), requests=rng.randint(3, 12),
                    reads=_log_int(rng, 10_000, 150_000))
    if what == "index":
        return dict(task="index", genome=rng.choice(["uniform", "adna", "genome"]), bp=_log_int(rng, 100_000, 100_000_000))
    return dict(task="pos", genome="adna", bp=_log_int(rng, 5_000_000, 100_000_000), rows=_log_int(rng, 1_000, 2_000_000))


# ---------------------------------------------------------------------------------------------------------------
# genomes

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _bases(n, g, gc=0.5):
    """n base codes (0..3 = A, C, G, T) with the given G + C share."""
    u = torch.rand(n, generator=g, device="cuda")
    return ((u > (1 - gc) / 2).to(torch.uint8) + (u > 0.5).to(torch.uint8) + (u > (1 + gc) / 2).to(torch.uint8))


def _diverged(codes, g, rate):
    hit = torch.rand(codes.shape, generator=g, device="cuda") < rate
    step = torch.randint(1, 4, codes.shape, generator=g, device="cuda", dtype=torch.uint8)
    return torch.where(hit, (codes + step) & 3, codes)


def _place(text, where, unit, copies):
    """copies (m x unit) at m distinct slots of `unit` bases."""
    slots = text[:len(text) // unit * unit].view(-1, unit)
    slots[where] = copies


def _strands(copies, g):
    rev = torch.rand(len(copies), generator=g, device="cuda") < 0.5
    return torch.where(rev[:, None], 3 - copies.flip(1), copies)


def _genome_text(kind, bp, seed):
    """The forward sequence (codes 0..3, on the GPU) of a reference of the workloads' kinds."""
    g = _generator(seed)
    if kind == "uniform":
        return _bases(bp, g)
    if kind == "adna":   # 45% GC, 5% in copies of 300 bp families at 10% divergence
        text = _bases(bp, g, 0.45)
        fam = _bases(50 * 300, g, 0.45).view(50, 300)
        where = torch.randperm(bp // 300, generator=g, device="cuda")[:int(0.05 * bp / 300)]
        of = torch.randint(0, 50, (len(where),), generator=g, device="cuda")
        _place(text, where, 300, _strands(_diverged(fam[of], g, 0.10), g))
        return text
    # genome: 25% 6 kbp copies at 8%, 20% 300 bp copies at 15%, 5% tandem repeats of 2-50 bp units at 2%
    text = _bases(bp, g, 0.41)
    long_n = int(0.25 * bp / 6000)
    where = torch.randperm(bp // 6000, generator=g, device="cuda")
    fam = _bases(5 * 6000, g, 0.40).view(5, 6000)
    for part in torch.split(where[:long_n], 2048):
        of = torch.randint(0, 5, (len(part),), generator=g, device="cuda")
        _place(text, part, 6000, _strands(_diverged(fam[of], g, 0.08), g))
    short = (where[long_n:, None] * 20 + torch.arange(20, device="cuda")).reshape(-1)   # 300 bp slots outside them
    short = short[torch.randperm(len(short), generator=g, device="cuda")]
    alu_n, tan_n = int(0.20 * bp / 300), int(0.05 * bp / 300)
    fam = _bases(20 * 300, g, 0.52).view(20, 300)
    for part in torch.split(short[:alu_n], 1 << 16):
        of = torch.randint(0, 20, (len(part),), generator=g, device="cuda")
        _place(text, part, 300, _strands(_diverged(fam[of], g, 0.15), g))
    for part in torch.split(short[alu_n:alu_n + tan_n], 1 << 16):
        unit = _bases(len(part) * 50, g).view(-1, 50)
        ulen = torch.randint(2, 51, (len(part), 1), generator=g, device="cuda")
        _place(text, part, 300, _diverged(unit.gather(1, torch.arange(300, device="cuda") % ulen), g, 0.02))
    return text


class _Genome:
    """A reference sequence with its resident indexes (one handle per trace setting) and its server."""

    def __init__(self, kind, bp):
        self.text = _genome_text(kind, bp, 1)
        self.handles, self.serving = {}, None
        with tempfile.TemporaryDirectory() as d:
            prefix = os.path.join(d, "ref")
            galn_b200.index_text(self.text.cpu().numpy(), prefix)
            for trace in (False, True):
                ix = galn_b200.Index(prefix)
                ix.set_trace(trace)
                self.handles[trace] = ix
            self.handles[False].load_sa(prefix)

    def server(self):
        if self.serving is None:
            self.serving = galn_b200.Server(self.handles[False])
        return self.serving

    def close(self):
        if self.serving is not None:
            self.serving.close()
        for ix in self.handles.values():
            ix.close()


_genomes: OrderedDict = OrderedDict()


def _genome(kind, bp):
    key = (kind, bp)
    if key not in _genomes:
        while len(_genomes) >= 2:
            _genomes.popitem(last=False)[1].close()
        _genomes[key] = _Genome(kind, bp)
    _genomes.move_to_end(key)
    return _genomes[key]


# ---------------------------------------------------------------------------------------------------------------
# reads

_ASCII = np.frombuffer(b"ACGTN", np.uint8)


def _lengths(kind, n, length, g):
    if kind == "adna":   # log-normal, mean 50, 25-120 bp
        sigma = 0.45
        z = torch.randn(n, generator=g, device="cuda")
        return torch.exp(z * sigma + (math.log(50) - sigma * sigma / 2)).round().clamp(25, 120).long()
    if kind in ("mixed", "mixed_adna"):
        return torch.randint(36, 151, (n,), generator=g, device="cuda")
    return torch.full((n,), length, dtype=torch.long, device="cuda")


def _reads_part(text, kind, lens, g):
    """Base codes (0..4) of reads drawn from both strands of the text, with the kind's errors."""
    n, width = len(lens), int(lens.max())
    j = torch.arange(width, device="cuda")
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda")   # noqa: E731
    pos = (rand(n).double() * (len(text) - 2 * width - 8)).long()
    off = j.expand(n, width)
    indel = dict(plain=0.001, divergent=0.005, genome=0.0005).get(kind, 0.0)
    inserted = None
    if indel:   # at most one insertion or deletion of 1-3 bp in a read
        has = rand(n) < indel * lens
        at = (1 + rand(n) * (lens - 2)).long()[:, None]
        size = torch.randint(1, 4, (n, 1), generator=g, device="cuda")
        is_del = (rand(n) < 0.5)[:, None]
        past = (j - at + 1).clamp(min=0)
        inserted = has[:, None] & ~is_del & (past > 0) & (past <= size)
        off = off + torch.where(has[:, None], torch.where(is_del, (past > 0) * size, -torch.minimum(past, size)), 0)
    rev = (rand(n) < 0.5)[:, None]
    span = (lens + 4)[:, None]
    codes = text[pos[:, None] + torch.where(rev, span - 1 - off, off)]
    codes = torch.where(rev, 3 - codes, codes)
    if inserted is not None:
        codes = torch.where(inserted, _bases(n * width, g).view(n, width), codes)
    rel = j / (lens[:, None] - 1)
    sub = {"plain": 0.01, "adna": 0.005, "mixed": 0.01, "mixed_adna": 0.005, "divergent": 0.04}.get(kind)
    rate = 0.001 + 0.014 * rel if sub is None else sub
    step = torch.randint(1, 4, (n, width), generator=g, device="cuda", dtype=torch.uint8)
    codes = torch.where(rand(n, width) < rate, (codes + step) & 3, codes)
    if kind in ("adna", "mixed_adna"):   # C->T at the 5' end, G->A at the 3' end
        codes = torch.where((codes == 1) & (rand(n, width) < 0.3 * 0.5 ** j), 3, codes)
        codes = torch.where((codes == 2) & (rand(n, width) < 0.3 * 0.5 ** (lens[:, None] - 1 - j)), 0, codes)
    strangers = dict(plain=0.02, adna=0.03, mixed=0.03, mixed_adna=0.03).get(kind, 0.0)
    codes = torch.where((rand(n) < strangers)[:, None], _bases(n * width, g).view(n, width), codes)
    if kind == "genome":   # reads that reach into a run of Ns of the reference
        codes = torch.where((rand(n) < 0.003)[:, None] & (j < rand(n)[:, None] * lens[:, None]), 4, codes)
    return codes[j < lens[:, None]]


def _reads(text, kind, n, length, seed):
    g = _generator(seed)
    lens = _lengths(kind, n, length, g)
    codes = torch.cat([_reads_part(text, kind, part, g) for part in torch.split(lens, 1 << 17)])
    off = torch.zeros(n + 1, dtype=torch.long, device="cuda")
    off[1:] = torch.cumsum(lens, 0)
    return galn_b200.Reads(_ASCII[codes.cpu().numpy()], off.cpu().numpy())


# ---------------------------------------------------------------------------------------------------------------

def _request_sizes(case):
    """Log-uniform sizes from a hundredth of the largest on, which is a quarter of the burst's reads."""
    k = case["requests"]
    w = [math.exp(math.log(0.01) * ((7 * i) % k) / max(1, k - 1)) for i in range(k)]
    return [max(1, int(case["reads"] * x / sum(w))) for x in w]


def prepare(case, seed):
    task = case["task"]
    if task == "index":
        d = tempfile.TemporaryDirectory()
        fwd = _genome_text(case["genome"], case["bp"], 1_000_003 + seed).cpu().numpy()
        return dict(task=task, fwd=fwd, dir=d, prefix=os.path.join(d.name, "ref"))
    ref = _genome(case["genome"], case["bp"])
    if task == "aln":
        reads = _reads(ref.text, case["kind"], case["reads"], case["length"], seed)
        return dict(task=task, index=ref.handles[case["trace"]], opts=galn_b200.parse_options(KINDS[case["kind"]]["opts"]),
                    reads=reads, trace=case["trace"], space=_record_space(case["reads"]))
    if task == "serve":
        requests = []
        for i, n in enumerate(_request_sizes(case)):
            kind = "mixed_adna" if i % 2 else "mixed"
            requests.append((galn_b200.parse_options(KINDS[kind]["opts"]),
                             _reads(ref.text, kind, n, 0, 64 * seed + i)))
        return dict(task=task, server=ref.server(), requests=requests, space=[_record_space(len(r)) for _, r in requests])
    g = _generator(seed)
    rows = torch.randint(1, 2 * case["bp"] + 1, (case["rows"],), generator=g, device="cuda")
    span = torch.randint(25, 121, (case["rows"],), generator=g, device="cuda", dtype=torch.int32)
    return dict(task=task, index=ref.handles[False], rows=rows.cpu().numpy().astype(np.uint64), span=span.cpu().numpy())


def _record_space(n):
    """Room for the records of n reads (about one a read), kept by the program, and how many it holds."""
    return dict(buf=np.zeros((2 * n + 4096, 3), np.int64), held=0)


def _arrays(res, trace, space):
    """The results, the records gathered into the program's own space (zeros past them)."""
    k, buf = len(res.records), space["buf"]
    buf[:k] = res.records.view(np.int64).reshape(k, 3)
    buf[k:space["held"]] = 0
    space["held"] = k
    out = dict(n_aln=res.n_aln, rec_offset=res.rec_offset, records=buf, pops=res.pops.view(np.int64))
    if trace:
        out["trace"] = res.trace.view(np.int64)
    return out


def run(state):
    task = state["task"]
    if task == "aln":
        return _arrays(galn_b200.aln(state["index"], state["opts"], state["reads"]), state["trace"], state["space"])
    if task == "serve":
        server = state["server"]
        ids = [server.submit(opts, reads) for opts, reads in state["requests"]]
        return [_arrays(server.wait(i), False, space) for i, space in zip(ids, state["space"])]
    if task == "index":
        galn_b200.index_text(state["fwd"], state["prefix"])
        return [np.memmap(state["prefix"] + ext, np.uint8, "r") for ext in (".bwt", ".sa")]
    pos, strand = state["index"].sa2pos(state["rows"], state["span"])
    return pos.view(np.int64), strand


def work(case):
    task, text = case["task"], 2 * case["bp"]
    index = text // 2
    if task == "index":   # the sequence in, the .bwt (2 bits a symbol and counts) and .sa (8 bytes in 32) out
        return dict(bytes=case["bp"] + text // 2 + text // 4, flops=text * math.log2(text))
    if task == "pos":     # a walk of 16 steps on average
        blocks = 16 * case["rows"]
        return dict(bytes=21 * case["rows"] + min(index, 32 * blocks), flops=OPS_PER_BLOCK * blocks / 4)
    if task == "serve":
        parts = [(n, 93, KINDS["mixed_adna" if i % 2 else "mixed"]["blocks"]) for i, n in enumerate(_request_sizes(case))]
    else:
        length = case["length"] or (50 if case["kind"] == "adna" else 93)
        parts = [(case["reads"], length, KINDS[case["kind"]]["blocks"])]
    blocks = sum(n * b for n, _, b in parts)
    # bases and offsets in; n_aln, record offset, pops and about one record out; each index block once
    return dict(bytes=sum(n * (length + 8 + 20 + 24) for n, length, _ in parts) + min(index, 32 * blocks),
                flops=OPS_PER_BLOCK * blocks)


def tolerance(case):
    return "exact"
