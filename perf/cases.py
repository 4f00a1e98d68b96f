"""Work that a user of rabbitbin_b200 has it do, as timed cases.

Every case goes through the public entry points of ``rabbitbin_b200.api`` on a
seeded synthetic assembly with the shapes and value laws of the package's own
workloads (``rabbitbin_b200.synth`` and ``rabbitbin_b200.workloads``): order-3
Markov genomes, log-normal contig lengths (median 6 kb, sigma 0.8, clipped to
2,500..80,000), one genome per 500 contigs (10 to 300), log-normal genome x
sample coverage with Poisson contig means.  Bases are drawn on the GPU, so
that preparing a large assembly takes about a second.

Kinds of case:

* ``bin``       contigs and coverage in host memory -> weighted graph (one call);
* ``resident``  the same on inputs staged on the device (repeated runs on one
                assembly), the graph fetched back;
* ``fasta``     the bytes of a FASTA file -> weighted graph;
* ``batch``     many assemblies of uneven sizes in one call;
* ``labels``    the weighted graph -> bins (Fisher label propagation);
* ``depth``     BAM files -> coverage matrix;
* ``winners``   contigs -> ProbMinHash winner rows (the sketch alone);
* ``compare``   sketch rows against sketch rows (many-vs-many queries).
"""
import ctypes
import math

import numpy as np
import torch

from rabbitbin_b200 import api
from rabbitbin_b200.synth import BAM_CLEAN, make_bam

SEG = 512                    # bases drawn in one chain on the GPU
_handle = []


def _context():
    """The one context that a program keeps for its calls."""
    if not _handle:
        _handle.append(api.Context(0))
    return _handle[0]


# ── inputs ─────────────────────────────────────────────────────────────────
def _genomes_for(n):
    return int(min(300, max(10, n // 500)))


def _offsets(rng, n):
    lens = np.exp(rng.normal(np.log(6000.0), 0.8, size=n))
    offs = np.zeros(n + 1, np.int64)
    np.cumsum(np.clip(lens, 2500, 80000).astype(np.int64), out=offs[1:])
    return offs


def _bases(rng, gen, offs, genome_of, n_genomes):
    """ASCII bases of every contig back to back (device uint8): one order-3
    chain of its genome per 512 bases, and a run of N per 2 Mbp."""
    dev = torch.device("cuda")
    p = rng.dirichlet(np.full(4, 0.5), size=(n_genomes, 64))
    gc = rng.uniform(-0.9, 0.9, size=(n_genomes, 1, 1))
    p = np.maximum(p, 1e-6) * np.exp(gc * np.array([0.0, 1.0, 1.0, 0.0]))
    cum = np.cumsum(p / p.sum(axis=2, keepdims=True), axis=2)[:, :, :3]
    cum = torch.from_numpy(cum.reshape(-1, 3).astype(np.float32)).to(dev)
    total = int(offs[-1])
    ends = torch.from_numpy(offs[1:]).to(dev)
    genome = torch.from_numpy(genome_of.astype(np.int64)).to(dev)
    nseg = -(-total // SEG)
    start = torch.arange(nseg, device=dev) * SEG
    contig = torch.searchsorted(ends, start, right=True).clamp_(max=len(genome_of) - 1)
    left = ends[contig] - start                      # bases until the next contig
    row = genome[contig] * 64
    state = torch.randint(0, 64, (nseg,), device=dev, generator=gen)
    out = torch.empty((SEG, nseg), dtype=torch.uint8, device=dev)
    for i in range(SEG):
        u = torch.rand(nseg, device=dev, generator=gen)
        base = (u[:, None] >= cum[row + state]).sum(dim=1)
        out[i] = base
        state = ((state << 2) | base) & 63
        if i % 64 == 63 and i + 1 < SEG:             # a segment that runs into its next contig
            left -= 64
            contig = torch.where(left <= 0, contig + 1, contig).clamp_(max=len(genome_of) - 1)
            left = ends[contig] - start - (i + 1)
            row = genome[contig] * 64
    seq = torch.empty(nseg * SEG, dtype=torch.uint8, device=dev)
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=dev)
    step = max(1, (1 << 27) // SEG)
    for s in range(0, nseg, step):
        part = out[:, s:s + step].t().reshape(-1)
        seq[s * SEG:s * SEG + part.numel()] = letters[part.int()]
    seq = seq[:total]
    runs = total // 2_000_000
    if runs:
        at = torch.from_numpy(rng.integers(0, total - 64, size=runs)).to(dev)
        width = torch.from_numpy(rng.integers(1, 60, size=runs)).to(dev)
        k = torch.arange(60, device=dev)
        seq[(at[:, None] + k)[k < width[:, None]]] = ord("N")
    return seq


def _coverage(rng, gen, genome_of, n_genomes, S):
    mean = np.exp(rng.normal(2.0, 1.0, size=(n_genomes, S))).astype(np.float32)
    rate = torch.from_numpy(mean).cuda()[torch.from_numpy(genome_of).cuda()]
    return torch.poisson(rate, generator=gen).cpu()


def _assembly(n, S, seed):
    """(ASCII bases on the device, offsets, coverage) of one assembly."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = _genomes_for(n)
    genome_of = rng.integers(0, g, size=n)
    offs = _offsets(rng, n)
    return _bases(rng, gen, offs, genome_of, g), offs, _coverage(rng, gen, genome_of, g, S)


class _Host:
    """An assembly in pinned host memory, as the API takes it."""

    def __init__(self, n, S, seed):
        seq, self.offsets, depth = _assembly(n, S, seed)
        self.seq = torch.empty(seq.numel(), dtype=torch.uint8, pin_memory=True)
        self.seq.copy_(seq)
        self.depth_pin = depth.contiguous().pin_memory()
        self.depth = self.depth_pin.numpy()
        self.ptr = ctypes.cast(ctypes.c_void_p(self.seq.data_ptr()), ctypes.c_char_p)


def _fasta(n, S, seed):
    """(pinned FASTA bytes, coverage): 80 bases a line, `>contig_<i>` headers."""
    seq, offs, depth = _assembly(n, S, seed)
    lens = np.diff(offs)
    head = [f">contig_{i}\n".encode() for i in range(n)]
    hlen = np.array([len(h) for h in head])
    lines = -(-lens // 80)
    first = np.zeros(n + 1, np.int64)
    np.cumsum(hlen + lens + lines, out=first[1:])
    out = torch.full((int(first[-1]),), ord("\n"), dtype=torch.uint8, device="cuda")
    body = torch.from_numpy(first[:-1] + hlen).cuda()
    off = torch.from_numpy(offs).cuda()
    step = 1 << 27
    for a in range(0, seq.numel(), step):
        q = torch.arange(a, min(a + step, seq.numel()), device="cuda")
        c = torch.searchsorted(off[1:], q, right=True)
        q -= off[c]
        out[body[c] + q + q // 80] = seq[a:a + step]
    hat = np.repeat(first[:-1] - np.concatenate([[0], np.cumsum(hlen)[:-1]]), hlen)
    hat += np.arange(len(hat))
    out[torch.from_numpy(hat).cuda()] = torch.from_numpy(
        np.frombuffer(b"".join(head), np.uint8).copy()).cuda()
    pin = torch.empty(out.numel(), dtype=torch.uint8, pin_memory=True)
    pin.copy_(out)
    return pin, depth.numpy()


def _batch_sizes(case):
    """(n, S, m) of each assembly of a batch: the mixed stream's law.  They
    belong to the case, not to the seed, so that its work is known."""
    rng = np.random.default_rng(case["mix"])
    n = np.exp(rng.uniform(np.log(case["n_min"]), np.log(case["n_max"]), size=case["count"]))
    S = rng.choice([3, 5, 10, 30], size=case["count"])
    m = rng.choice([250, 500, 1000], size=case["count"])
    return [(int(a), int(b), int(c)) for a, b, c in zip(n, S, m)]


def _sketch_rows(case, seed, dtype):
    """Query and target sketch rows: 200 related groups, a member keeps each
    register of its group with a probability of its own."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m, n = case["m"], case["na"] + case["nb"]
    group = torch.randint(0, 200, (n,), device="cuda", generator=gen)
    if dtype == "registers":
        def draw(k):
            return -torch.log1p(-torch.rand((k, m), device="cuda", generator=gen,
                                            dtype=torch.float64))
    else:
        def draw(k):
            return torch.randint(1, 2**62, (k, m), device="cuda", generator=gen)
    base = draw(200)[group]
    own = draw(n)
    keep = torch.rand((n, m), device="cuda", generator=gen) < torch.rand(
        (n, 1), device="cuda", generator=gen)
    rows = torch.where(keep, base, own).cpu().numpy()
    if dtype != "registers":
        rows = rows.view(np.uint64)
    return rows[:case["na"]], rows[case["na"]:]


# ── the cases ──────────────────────────────────────────────────────────────
def listed():
    return [
        # the smallest call: a single-sample isolate-like assembly, all latency
        {"name": "bin_97_s1", "kind": "bin", "n": 97, "S": 1, "m": 500},
        # a small metagenome in one call (small path, every pair compared)
        {"name": "bin_2000_s5", "kind": "bin", "n": 2000, "S": 5, "m": 500},
        # repeated runs on a mid-size assembly: the dense regime below 25,000 contigs
        {"name": "resident_20011_s5", "kind": "resident", "n": 20011, "S": 5, "m": 500},
        # the binning-scale assembly on staged inputs: the abundance-pruned regime
        {"name": "resident_50000_s20", "kind": "resident", "n": 50000, "S": 20, "m": 500},
        # a large many-sample assembly in one call from host memory
        {"name": "bin_200003_s30", "kind": "bin", "n": 200003, "S": 30, "m": 500},
        # a file's bytes to the graph, few samples (the prune passes many pairs)
        {"name": "fasta_30011_s5", "kind": "fasta", "n": 30011, "S": 5, "m": 500},
        # a mixed stream of assemblies in one call
        {"name": "batch_16", "kind": "batch", "count": 16, "n_min": 1000, "n_max": 40000,
         "mix": 3},
        # graph -> bins, the default sequential sweep, and the synchronous one
        {"name": "labels_50000", "kind": "labels", "n": 50000, "S": 20, "sync": False},
        {"name": "labels_sync_20011", "kind": "labels", "n": 20011, "S": 10, "sync": True},
        # BAM files of two samples -> coverage
        {"name": "depth_8000_x2", "kind": "depth", "n": 8000, "bams": 2, "cover": 1.5},
        # the sketch alone, wide rows
        {"name": "winners_5003_m1000", "kind": "winners", "n": 5003, "m": 1000, "k": 4},
        # queries against a sketch collection
        {"name": "compare_1000x4999", "kind": "compare", "na": 1000, "nb": 4999, "m": 500,
         "metric": "distance"},
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["bin", "bin", "resident", "resident", "fasta", "batch", "labels",
                       "depth", "winners", "compare"])
    m = rng.choice([250, 500, 1000])
    if kind == "bin":
        return {"kind": kind, "n": span(50, 120000), "S": rng.choice([5, 10, 20, 30]), "m": m}
    if kind == "resident":
        return {"kind": kind, "n": span(500, 80000), "S": rng.choice([3, 5, 10, 20, 30]), "m": m}
    if kind == "fasta":
        return {"kind": kind, "n": span(300, 60000), "S": rng.choice([3, 5, 10, 20]), "m": m}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 14), "n_min": 500, "n_max": 30000,
                "mix": rng.randrange(1 << 20)}
    if kind == "labels":
        return {"kind": kind, "n": span(500, 60000), "S": rng.choice([5, 10, 20]),
                "sync": rng.random() < 0.4}
    if kind == "depth":
        return {"kind": kind, "n": span(100, 12000), "bams": rng.randint(1, 3),
                "cover": round(rng.uniform(0.5, 1.5), 2)}
    if kind == "winners":
        return {"kind": kind, "n": span(50, 30000), "m": m, "k": rng.choice([3, 4, 4])}
    return {"kind": kind, "na": span(10, 2000), "nb": span(100, 8000), "m": m,
            "metric": rng.choice(["jaccard_weighted", "jaccard", "distance", "ani"])}


class _Edges:
    """A program's own edge arrays on the GPU (for its next step), sized for
    the most edges that 200 neighbours a contig can give (100 a contig where
    the lists have to be mutual, above 25,000 contigs); entries past the last
    edge are 0."""

    def __init__(self, ns):
        cap = sum(min((100 if n > 25000 else 200) * n, n * (n - 1) // 2) for n in ns)
        kinds = {"src": torch.int32, "dst": torch.int32, "scomp": torch.float32,
                 "score": torch.float32}
        self.arrays = {k: torch.zeros(cap, dtype=t, device="cuda") for k, t in kinds.items()}
        self.used = 0

    def take(self, graphs):
        at = 0
        for g in graphs:
            e = len(g["src"])
            for k, to in self.arrays.items():
                a = g[k].view(np.int32) if to.dtype == torch.int32 else g[k]
                to[at:at + e].copy_(torch.from_numpy(a))
            at += e
        if at < self.used:
            for to in self.arrays.values():
                to[at:self.used].zero_()
        self.used = at
        return dict(self.arrays, n_edges=np.array([len(g["src"]) for g in graphs]),
                    b0=np.array([g["b0"] for g in graphs]),
                    sim_cutoff=np.array([g["sim_cutoff"] for g in graphs]))


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case, "ctx": _context()}
    if kind in ("bin", "resident"):
        a = _Host(case["n"], case["S"], seed)
        st["params"] = api.default_params(m=case["m"])
        if kind == "bin":
            st["asm"] = a
        else:                                        # staged inputs live in a context of their own
            st["ctx"] = api.Context(0)
            st["ctx"].stage(a.ptr, a.offsets, a.depth)
    elif kind == "fasta":
        st["data"], st["depth"] = _fasta(case["n"], case["S"], seed)
        st["ptr"] = ctypes.cast(ctypes.c_void_p(st["data"].data_ptr()), ctypes.c_char_p)
        st["params"] = api.default_params(m=case["m"])
    elif kind == "batch":
        st["hosts"] = [_Host(n, S, seed * 1009 + i)
                       for i, (n, S, _) in enumerate(_batch_sizes(case))]
        st["asms"] = [(h.ptr, h.offsets, h.depth, api.default_params(m=m))
                      for h, (_, _, m) in zip(st["hosts"], _batch_sizes(case))]
    elif kind == "labels":
        a = _Host(case["n"], case["S"], seed)
        g = st["ctx"].bin_graph(a.ptr, a.offsets, a.depth)
        st["graph"] = tuple(g[k].copy() for k in ("src", "dst", "score"))
    elif kind == "depth":
        n = case["n"]
        seq, offs, depth = _assembly(n, case["bams"], seed)
        host = seq.cpu().numpy()
        lens = np.diff(offs).astype(np.uint32)
        cov = depth.numpy().astype(np.float64)
        cov *= case["cover"] / np.maximum(cov.mean(axis=0), 1e-9)
        st["bams"] = [make_bam(lens, cov[:, b], seq=host, seq_off=offs, seed=seed * 31 + b,
                               read_len=150, level=6, **BAM_CLEAN) for b in range(case["bams"])]
    elif kind == "winners":
        st["asm"] = _Host(case["n"], 0, seed)
        st["params"] = api.default_params(m=case["m"], k=case["k"])
    else:
        st["rows"] = _sketch_rows(case, seed, "winners" if case["metric"] == "jaccard_weighted"
                                  else "registers")
    if kind in ("bin", "resident", "fasta"):
        st["edges"] = _Edges([case["n"]])
    elif kind == "batch":
        st["edges"] = _Edges([n for n, _, _ in _batch_sizes(case)])
    return st


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "bin":
        a = state["asm"]
        return state["edges"].take([ctx.bin_graph(a.ptr, a.offsets, a.depth, state["params"])])
    if kind == "resident":
        ctx.run_resident(state["params"])
        return state["edges"].take([ctx.fetch_graph()])
    if kind == "fasta":
        return state["edges"].take([ctx.bin_fasta(state["ptr"], state["depth"],
                                                  params=state["params"],
                                                  nbytes=state["data"].numel())])
    if kind == "batch":
        graphs, _ = ctx.bin_batch(state["asms"])
        return state["edges"].take(graphs)
    if kind == "labels":
        src, dst, score = state["graph"]
        labels, _ = ctx.label_propagation(state["case"]["n"], src, dst, score, seed=1,
                                          rule="fisher", synchronous=state["case"]["sync"])
        return labels.view(np.int32)
    if kind == "depth":
        d = ctx.bam_depth(state["bams"])
        return {"tid": d["tid"], "lens": d["lens"], "means": d["means"],
                "sums": d["sums"].view(np.int64), "avg_read": d["avg_read"]}
    if kind == "winners":
        a = state["asm"]
        return ctx.build_pmh_winners(a.ptr, a.offsets, state["params"]).view(np.int32)
    A, B = state["rows"]
    return ctx.pmh_compare(state["case"]["metric"], A, B, 4)


# ── what a pass cannot do without ──────────────────────────────────────────
def _bases_of(n):
    """Expected bases of n contigs (the clipped log-normal's mean)."""
    return 8360.0 * n


def _bin_work(n, S, m, edges=50.0):
    """Bases and coverage in, about 50 edges a contig out; per unordered pair
    the smaller of the two tests the path knows: the rank-correlation product
    of 2 S operations (many samples) or m register compares (below 25,001
    contigs, where nothing is pruned)."""
    pairs = 0.5 * n * (n - 1.0)
    per_pair = 2.0 * S if n > 25000 and S > 2 else float(m)
    return {"bytes": _bases_of(n) + 4.0 * n * S + 16.0 * edges * n, "flops": pairs * per_pair}


def work(case):
    kind = case["kind"]
    if kind in ("bin", "resident", "fasta"):
        return _bin_work(case["n"], case["S"], case["m"])
    if kind == "batch":
        parts = [_bin_work(*s) for s in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "labels":                             # 12 bytes an edge, every arc read once
        return {"bytes": 50.0 * case["n"] * (12.0 + 16.0), "flops": 0.0}
    if kind == "depth":                              # reads of about 300 bytes, compressed to 48
        reads = case["cover"] * _bases_of(case["n"]) / 150.0 * case["bams"]
        return {"bytes": reads * (48.0 + 300.0), "flops": 0.0}
    if kind == "winners":
        return {"bytes": _bases_of(case["n"]) + 4.0 * case["n"] * case["m"], "flops": 0.0}
    na, nb, m = case["na"], case["nb"], case["m"]
    return {"bytes": 8.0 * ((na + nb) * m + na * nb), "flops": float(na) * nb * m}


def exact(case, seed):
    """Query values in 64 bits.  A graph's weights, a BAM's means and labels
    follow from whole-number decisions along the path (register winners, read
    filters) that plain array code has no short form of."""
    if case["kind"] != "compare":
        return None
    A, B = _sketch_rows(case, seed, "winners" if case["metric"] == "jaccard_weighted"
                        else "registers")
    m = case["m"]
    a = torch.from_numpy(A.view(np.int64).copy()).cuda()
    b = torch.from_numpy(B.view(np.int64).copy()).cuda()
    out = torch.empty((len(A), len(B)), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 28) // (len(B) * m))
    for s in range(0, len(A), step):
        out[s:s + step] = (a[s:s + step, None, :] == b[None]).sum(dim=2).double() / m
    if case["metric"] in ("distance", "ani"):
        mash = 2.0 * out / (1.0 + out)
        if case["metric"] == "distance":
            out = -torch.log(mash) / 4.0                  # +inf without a common register
        else:
            out = mash ** 0.25
    return out.cpu().numpy()
