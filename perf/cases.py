"""The work that a user of this framework has it do, as cases that can be timed.

A run of the framework on one assembly is: the FASTA file's record split, the
tetranucleotide count of every contig, the sampled search for the probability
cutoff, the all-pairs graph at that cutoff, the abundance scoring of its edges,
label propagation over them, and the recruiting of what was left out.  There is
a case for each of these calls, one for the three that the benchmark times as
one step, one for many small assemblies in a batch, and one for the training
of the learned proposal.  Sizes run from a draft genome's few hundred contigs
to the benchmark's million-contig assembly.

Assemblies are synthetic, as in the benchmark: genomes are order-3 Markov chains
with GC 0.3 to 0.7, contig lengths log-normal and clamped, 0.5 % N.  They are
made on the GPU here, since preparing a case makes several of them.
"""
from __future__ import annotations

import ctypes
import math
import statistics

import numpy as np
import torch

import mdet_gb300 as mdet

NTNF = 136


def listed():
    return [
        # one isolate's draft assembly, one sequence per line as some assemblers
        # write it: the smallest call, where launches and waits are all there is
        {"name": "count_draft_300", "kind": "count", "n": 300, "width": 0},
        # a large metagenome's sequences, 60 columns: the read of the whole file
        {"name": "count_400k", "kind": "count", "n": 400000, "width": 60},
        # the record split of a whole file, most records below the size limit
        {"name": "index_220k", "kind": "index", "n": 220007, "width": 80},
        # one pass of the cutoff search: 2,500 sampled contigs against all
        {"name": "sample_250k", "kind": "sample", "n": 250013, "m": 2500, "floor": 0.7},
        # the graph of a small sample: latency
        {"name": "graph_1500", "kind": "graph", "n": 1500, "mode": "bf16", "cutoff": 0.9, "max_edges": 200},
        # the graph in the TF32 form, at the size of the reference's first configuration
        {"name": "graph_tf32_20k", "kind": "graph", "n": 20011, "mode": "tf32", "cutoff": 0.909, "max_edges": 200},
        # the benchmark's step: count, cutoff search and graph of a million contigs
        {"name": "step_1m", "kind": "step", "n": 1000000, "max_edges": 200},
        # a study of many small assemblies, their graphs in one call
        {"name": "batch_48", "kind": "batch", "count": 48, "lo": 400, "hi": 6000, "cutoff": 0.9, "max_edges": 200},
        # the abundance scores of a graph's edges over ten samples
        {"name": "sscr_60k", "kind": "sscr", "n": 60000, "nabd": 10, "deg": 80},
        # binning by label propagation over the scored edges
        {"name": "labels_60k", "kind": "labels", "n": 60000, "deg": 60},
        # dissolving small bins and recruiting, through host arrays as the program holds them
        {"name": "recruit_150k", "kind": "recruit", "n": 150000, "small": 20000, "nabd": 10},
        # training the learned proposal (forward, backward, optimiser) on an assembly's pairs
        {"name": "train_20k", "kind": "train", "n": 20000, "pairs": 500000, "steps": 40, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count", "index", "sample", "graph", "graph", "step", "batch", "sscr", "labels", "recruit",
                       "train"])
    if kind == "count":
        return {"kind": kind, "n": _log_int(rng, 60, 400000), "width": rng.choice([0, 60, 61, 70, 80])}
    if kind == "index":
        return {"kind": kind, "n": _log_int(rng, 200, 220000), "width": rng.choice([0, 60, 61, 70, 80])}
    if kind == "sample":
        return {"kind": kind, "n": _log_int(rng, 3000, 300000), "m": rng.randint(500, 2500),
                "floor": rng.choice([0.7, 0.7, 0.85, 0.9])}
    if kind == "graph":
        mode = rng.choice(["bf16", "bf16", "bf16", "tf32"])
        return {"kind": kind, "n": _log_int(rng, 300, 250000 if mode == "bf16" else 80000), "mode": mode,
                "cutoff": rng.randint(800, 970) / 1000, "max_edges": rng.choice([30, 100, 200, 200, 400])}
    if kind == "step":
        return {"kind": kind, "n": _log_int(rng, 26000, 400000), "max_edges": rng.choice([100, 200])}
    if kind == "batch":
        lo = _log_int(rng, 200, 1000)
        return {"kind": kind, "count": rng.randint(4, 64), "lo": lo, "hi": _log_int(rng, 2 * lo, 9000),
                "cutoff": rng.randint(850, 960) / 1000, "max_edges": rng.choice([50, 200])}
    if kind == "sscr":
        return {"kind": kind, "n": _log_int(rng, 1500, 90000), "nabd": rng.randint(1, 16), "deg": rng.randint(20, 100)}
    if kind == "labels":
        return {"kind": kind, "n": _log_int(rng, 1000, 100000), "deg": rng.randint(15, 80)}
    if kind == "recruit":
        n = _log_int(rng, 3000, 250000)
        return {"kind": kind, "n": n, "small": rng.randint(1, n // 4), "nabd": rng.randint(3, 30)}
    return {"kind": "train", "n": _log_int(rng, 4000, 40000), "pairs": _log_int(rng, 50000, 1000000),
            "steps": rng.randint(15, 50), "batch": rng.choice([1024, 3000, 4096, 8192])}


# ------------------------------------------------------------- assemblies --

def _gen(case, seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt * 7919 + sum(case["kind"].encode())) % (1 << 62))
    return g


def _genomes(n):
    return max(3, n // 450)


def _assembly(g, n, genomes, width, median=5000.0, lo=2500, hi=500000):
    """FASTA bytes and sequence views of n contigs on the GPU.  width 0: one
    line per sequence.  Returns a dict of buf, nbytes, off, len, size, log_size,
    genome, name_off and name_len."""
    dev = "cuda"
    L = (torch.exp(torch.randn(n, generator=g, device=dev, dtype=torch.float64) + math.log(median))
         .clamp(lo, hi).floor().to(torch.int64))
    genome = torch.randint(0, genomes, (n,), generator=g, device=dev)
    # next-base thresholds of the 64 contexts of every genome
    gc = 0.3 + 0.4 * torch.rand(genomes, 1, generator=g, device=dev)
    base_p = torch.cat([(1 - gc) / 2, gc / 2, gc / 2, (1 - gc) / 2], 1)
    w = base_p[:, None, :] * torch.exp(0.25 * torch.randn(genomes, 64, 4, generator=g, device=dev))
    thr = (w.cumsum(2) / w.sum(2, keepdim=True))[:, :, :3].reshape(genomes * 64, 3).contiguous()
    # layout: ">ctg<k>\n", the sequence lines, each ended by a newline
    k = torch.arange(n, device=dev)
    digits = torch.ones_like(k)
    for d in range(1, 9):
        digits += (k >= 10 ** d).to(torch.int64)
    head = 5 + digits
    lines = torch.ones_like(L) if width == 0 else (L + width - 1) // width
    rec = head + L + lines
    end = rec.cumsum(0)
    start = end - rec
    nbytes = int(end[-1])
    buf = torch.full((nbytes + 64,), 10, dtype=torch.uint8, device=dev)
    for j, ch in enumerate(b">ctg"):
        buf[start + j] = ch
    for d in range(8):  # d-th digit from the right
        m = digits > d
        buf[(start + 4 + digits - 1 - d)[m]] = (48 + (k[m] // 10 ** d) % 10).to(torch.uint8)
    off = start + head
    # the bases: every contig in pieces of 256, each piece a lane of the chain
    C = 256
    acgtn = torch.tensor(list(b"ACGTN"), dtype=torch.uint8, device=dev)
    pieces = (L + C - 1) // C
    piece_end = pieces.cumsum(0)
    for c0 in range(0, int(piece_end[-1]), 1 << 24):
        lane = torch.arange(c0, min(c0 + (1 << 24), int(piece_end[-1])), device=dev)
        ctg = torch.searchsorted(piece_end, lane, right=True)
        pos = (lane - (piece_end - pieces)[ctg]) * C
        base, room = off[ctg], L[ctg]
        gen64 = (genome[ctg] * 64)
        ctx = torch.randint(0, 64, (lane.numel(),), generator=g, device=dev)
        for _ in range(C):
            r = torch.rand(lane.numel(), generator=g, device=dev)
            b = (r[:, None] >= thr[gen64 + ctx]).sum(1)
            ctx = ((ctx << 2) | b) & 63
            b = torch.where((r * 997).frac() < 0.005, 4, b)
            addr = base + pos if width == 0 else base + pos + pos // width
            addr = torch.where(pos < room, addr, nbytes + 32)
            buf[addr] = acgtn[b]
            pos += 1
    buf[nbytes:] = 10
    return {"buf": buf, "nbytes": nbytes, "off": off, "len": L + lines - 1, "size": L, "genome": genome,
            "log_size": torch.log10(L.clamp(max=500000).double()), "name_off": start + 1, "name_len": 3 + digits}


def _ptr(t):
    return t.data_ptr()


_shared = None


def _context():
    """The program's context: one for all its assemblies, on torch's stream."""
    global _shared
    if _shared is None:
        _shared = mdet.Context(0)
        _shared.set_stream(torch.cuda.current_stream().cuda_stream)
    return _shared


def _tnf(ctx, a):
    n = a["off"].numel()
    counts = torch.empty(n, NTNF, dtype=torch.int32, device="cuda")
    tnf = torch.empty(n, NTNF, dtype=torch.float32, device="cuda")
    ctx.tnf_count_dev(_ptr(a["buf"]), a["nbytes"], _ptr(a["off"]), _ptr(a["len"]), n, _ptr(counts), _ptr(tnf))
    return counts, tnf


def _rows(case, seed, n, salt=0):
    """TNF rows and log sizes of a counted assembly."""
    a = _assembly(_gen(case, seed, salt), n, _genomes(n), 60)
    _, tnf = _tnf(_context(), a)
    return tnf, a["log_size"]


def _edge_outputs(n, max_edges):
    # a contig keeps at most max_edges, and an edge is emitted once
    cap = n * min(max_edges, max(1, n - 1))
    return (torch.zeros(cap, dtype=torch.int64, device="cuda"), torch.zeros(cap, dtype=torch.int64, device="cuda"),
            torch.zeros(cap, dtype=torch.float64, device="cuda"))


def _depths(g, genome, nabd):
    """Mean depths and variances per contig and sample, shaped like a depth
    table: genome depths around 10x, contig noise, 3 % of contigs uncovered."""
    n, dev = genome.numel(), "cuda"
    gd = torch.exp(torch.randn(int(genome.max()) + 1, nabd, generator=g, device=dev, dtype=torch.float64)
                   + math.log(10.0))
    abd = gd[genome] * torch.exp(0.15 * torch.randn(n, nabd, generator=g, device=dev, dtype=torch.float64))
    low = torch.rand(n, generator=g, device=dev) < 0.03
    abd = torch.where(low[:, None], torch.rand(n, nabd, generator=g, device=dev, dtype=torch.float64), abd)
    var = abd * (0.5 + 1.5 * torch.rand(n, nabd, generator=g, device=dev, dtype=torch.float64))
    return abd.float().double(), var.float().double(), low


def _scored_edges(g, n, genomes, deg, keep=None):
    """Edges (from < to, by row) of a graph of n contigs, most of them within a
    genome, with scores as the graph gives them: high within, lower across."""
    dev = "cuda"
    genome = torch.randint(0, genomes, (n,), generator=g, device=dev)
    order = torch.argsort(genome, stable=True)
    count = torch.bincount(genome, minlength=genomes)
    first = count.cumsum(0) - count
    m = n * deg
    a = torch.randint(0, n, (m,), generator=g, device=dev)
    inside = torch.rand(m, generator=g, device=dev) < 0.85
    u = torch.rand(m, generator=g, device=dev, dtype=torch.float64)
    mate = order[(first[genome[a]] + (u * count[genome[a]]).long()).clamp(max=n - 1)]
    b = torch.where(inside, mate, (u * n).long().clamp(max=n - 1))
    ok = a != b
    if keep is not None:
        ok &= keep[a] | keep[b]
    lo, hi = torch.minimum(a, b)[ok], torch.maximum(a, b)[ok]
    key = torch.unique(lo * n + hi)
    # the same number of edges for every seed (a few are drawn twice)
    key = key[torch.randperm(key.numel(), generator=g, device=dev)[:int(0.8 * m)]].sort().values
    fr, to = key // n, key % n
    v = torch.rand(key.numel(), generator=g, device=dev, dtype=torch.float64)
    same = genome[fr] == genome[to]
    score = torch.where(same, 1 - 0.35 * v ** 1.5, 0.9 - 0.5 * v.sqrt())
    return genome, fr.contiguous(), to.contiguous(), score.contiguous()


# ---------------------------------------------------------------- prepare --

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case, "ctx": _context(), "seed": int(seed)}
    if kind in ("count", "step"):
        n = case["n"]
        a = _assembly(_gen(case, seed), n, _genomes(n), case.get("width", 60))
        s.update(a=a, counts=torch.empty(n, NTNF, dtype=torch.int32, device="cuda"),
                 tnf=torch.empty(n, NTNF, dtype=torch.float32, device="cuda"))
        if kind == "step":
            s["out"] = _edge_outputs(n, case["max_edges"])
            s["libc"] = ctypes.CDLL(None)  # the search draws from the C library's rand()
    elif kind == "index":
        n = case["n"]
        s["a"] = _assembly(_gen(case, seed), n, _genomes(n), case["width"], median=2500.0, lo=500)
        s["o64"] = [torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(4)]
        s["ls"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        s["o32"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif kind == "sample":
        n, m = case["n"], case["m"]
        s["tnf"], s["log_size"] = _rows(case, seed, n)
        s["contigs"] = torch.randperm(n, generator=_gen(case, seed, 1), device="cuda")
        s["out"] = torch.empty(m, dtype=torch.float64, device="cuda")
    elif kind == "graph":
        s["tnf"], s["log_size"] = _rows(case, seed, case["n"])
        s["out"] = _edge_outputs(case["n"], case["max_edges"])
    elif kind == "batch":
        sizes = _batch_sizes(case)
        s["sets"] = [_rows(case, seed, n, 100 + i) for i, n in enumerate(sizes)]
        s["caps"] = [n * min(case["max_edges"], n - 1) for n in sizes]
        s["out"] = [torch.zeros(sum(s["caps"]), dtype=t, device="cuda")
                    for t in (torch.int64, torch.int64, torch.float64)]
        s["items"], at = [], 0
        for (t, l), n, cap in zip(s["sets"], sizes, s["caps"]):
            o = [_ptr(x) + 8 * at for x in s["out"]]
            s["items"].append(dict(d_tnf=_ptr(t), d_ls=_ptr(l), n=n, cutoff=case["cutoff"],
                                   max_edges=case["max_edges"], d_from=o[0], d_to=o[1], d_stnf=o[2], capacity=cap))
            at += cap
    elif kind == "sscr":
        n, g = case["n"], _gen(case, seed)
        genome = torch.randint(0, _genomes(n), (n,), generator=g, device="cuda")
        abd, var, low = _depths(g, genome, case["nabd"])
        # an edge has a covered sample: the graph drops pairs of two uncovered contigs
        _, fr, to, st = _scored_edges(g, n, _genomes(n), case["deg"], keep=(abd > 1.0).any(1))
        # depths belong to an assembly, so it has a context of its own
        ctx = mdet.Context(0)
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        ctx.set_abundance(abd.cpu().numpy(), var.cpu().numpy())
        s.update(ctx=ctx, fr=fr, to=to, st=st, out=torch.empty_like(st), abd=abd, var=var)
    elif kind == "labels":
        _, s["fr"], s["to"], s["st"] = _scored_edges(_gen(case, seed), case["n"], _genomes(case["n"]), case["deg"])
        s["mem"] = torch.empty(case["n"], dtype=torch.int64, device="cuda")
    elif kind == "recruit":
        n, ns, g = case["n"], case["small"], _gen(case, seed)
        genome = torch.randint(0, _genomes(n), (n + ns,), generator=g, device="cuda")
        abd, _, _ = _depths(g, genome, case["nabd"])
        abd = abd.float().cpu().numpy()
        label = genome[:n].clone()
        tiny = torch.rand(n, generator=g, device="cuda") < 0.01
        label[tiny] = (1 << 40) + torch.arange(int(tiny.sum()), device="cuda")
        L = torch.exp(torch.randn(n, generator=g, device="cuda") + math.log(5000.0)).clamp(2500, 500000).long()
        small = torch.randint(1000, 2500, (ns,), generator=g, device="cuda")
        s.update(abd=np.ascontiguousarray(abd[:n]), sabd=np.ascontiguousarray(abd[n:]), label=label.cpu().numpy(),
                 sizes=L.cpu().numpy().astype(np.uint64), ssizes=small.cpu().numpy().astype(np.uint64))
    else:
        s["tnf"], s["log_size"] = _rows(case, seed, case["n"])
    return s


def _batch_sizes(case):
    # spread over the logarithm of the range, in an order that mixes them
    c = case["count"]
    r = [int(case["lo"] * (case["hi"] / case["lo"]) ** (((i * 29) % c + 0.5) / c)) | 1 for i in range(c)]
    return r


# -------------------------------------------------------------------- run --

def run(s):
    ctx, case, kind = s["ctx"], s["case"], s["kind"]
    if kind == "count":
        a = s["a"]
        ctx.tnf_count_dev(_ptr(a["buf"]), a["nbytes"], _ptr(a["off"]), _ptr(a["len"]), case["n"], _ptr(s["counts"]),
                          _ptr(s["tnf"]))
        return [s["counts"], s["tnf"]]
    if kind == "index":
        a, (off, ln, size, noff) = s["a"], s["o64"]
        st = ctx.fasta_index_dev(_ptr(a["buf"]), a["nbytes"], 2500, case["n"], _ptr(off), _ptr(ln), _ptr(size),
                                 _ptr(s["ls"]), _ptr(noff), _ptr(s["o32"]))
        return [st["n_records"], st["n_large"], st["n_small"], off, ln, size, s["ls"], noff, s["o32"]]
    if kind == "sample":
        ctx.max_prob_dev(_ptr(s["tnf"]), _ptr(s["log_size"]), case["n"], _ptr(s["contigs"]), case["m"], "bf16",
                         case["floor"], _ptr(s["out"]))
        # contigs with no pair at the floor report some value below it
        return [torch.where(s["out"] >= case["floor"], s["out"], 0.0)]
    if kind == "graph":
        fr, to, st = s["out"]
        k, _ = ctx.tnf_graph_dev(_ptr(s["tnf"]), _ptr(s["log_size"]), case["n"], case["cutoff"], case["max_edges"],
                                 case["mode"], _ptr(fr), _ptr(to), _ptr(st), fr.numel())
        return [k, fr, to, st]
    if kind == "step":
        a, n, (fr, to, st) = s["a"], case["n"], s["out"]
        ctx.tnf_count_dev(_ptr(a["buf"]), a["nbytes"], _ptr(a["off"]), _ptr(a["len"]), n, _ptr(s["counts"]),
                          _ptr(s["tnf"]))
        s["libc"].srand(s["seed"] % (1 << 31))
        ptnf = ctx.ptnf_search_dev(_ptr(s["tnf"]), _ptr(a["log_size"]), n, 0.95, "bf16")
        k, _ = ctx.tnf_graph_dev(_ptr(s["tnf"]), _ptr(a["log_size"]), n, ptnf / 1000.0, case["max_edges"], "bf16",
                                 _ptr(fr), _ptr(to), _ptr(st), fr.numel())
        return [s["counts"], s["tnf"], ptnf, k, fr, to, st]
    if kind == "batch":
        res, _ = ctx.tnf_graph_batched(s["items"], "bf16")
        return [sum(k for _, k in res)] + s["out"]
    if kind == "sscr":
        ctx.edges_sscr_dev(_ptr(s["fr"]), _ptr(s["to"]), _ptr(s["st"]), s["st"].numel(), _ptr(s["out"]))
        return [s["out"]]
    if kind == "labels":
        st = ctx.label_propagation_dev(_ptr(s["fr"]), _ptr(s["to"]), _ptr(s["st"]), s["st"].numel(), case["n"],
                                       _ptr(s["mem"]))
        return [s["mem"], st["calls"], st["sweeps"], st["connected"]]
    if kind == "recruit":
        out, sout, st = ctx.recruit(s["abd"], s["sabd"], s["label"], s["sizes"], s["ssizes"], 200000,
                                    int(s["ssizes"].sum()))
        return [out, sout, st["n_bins"], st["n_leftovers_matched"], st["n_small_matched"]]
    net = mdet.Network(ctx, s["seed"] % 1000 + 1)
    net.train_dev(_ptr(s["tnf"]), _ptr(s["log_size"]), case["n"], pairs=case["pairs"], steps=case["steps"],
                  batch_pairs=case["batch"])
    params = net.get_params()
    net.close()
    return [params]


# ------------------------------------------------------------------- work --

def _mean_size(median, lo, hi=500000.0):
    q = statistics.NormalDist()
    return sum(min(max(median * math.exp(q.inv_cdf((i + 0.5) / 4000)), lo), hi) for i in range(4000)) / 4000


def work(case):
    """What a pass cannot do without.  Contig lengths are drawn, so a file's
    bytes are their expected sum; so are the edges a graph keeps."""
    kind, n = case["kind"], case.get("n", 0)

    def text(median, lo):
        L, w = _mean_size(median, lo), case.get("width", 60)
        return n * (L + (L / w if w else 1) + 11)

    def graph(k, max_edges):
        kept = 0.3 * k * min(max_edges, 400, k)
        return {"bytes": k * (NTNF * 4 + 8) + 24 * kept, "flops": 136.0 * k * (k - 1)}

    if kind == "count":
        return {"bytes": text(5000.0, 2500) + n * (16 + 8 * NTNF), "flops": 0}
    if kind == "index":
        return {"bytes": text(2500.0, 500) + 0.5 * n * 44, "flops": 0}
    if kind == "sample":
        return {"bytes": n * (NTNF * 4 + 8) + 16 * case["m"], "flops": 2.0 * NTNF * n * case["m"]}
    if kind == "graph":
        return graph(n, case["max_edges"])
    if kind == "step":
        w = graph(n, case["max_edges"])
        m = 10 * 2500 * n if n > 25000 else n * n
        return {"bytes": text(5000.0, 2500) + n * (16 + 8 * NTNF) + w["bytes"], "flops": w["flops"] + 2.0 * NTNF * m}
    if kind == "batch":
        ws = [graph(k, case["max_edges"]) for k in _batch_sizes(case)]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    if kind == "sscr":
        ne, a = int(0.8 * n * case["deg"]), case["nabd"]
        # per edge and sample: two crossing points and four normal CDFs (about 100 operations in all)
        return {"bytes": 32.0 * ne + 16.0 * n * a, "flops": 100.0 * ne * a}
    if kind == "labels":
        return {"bytes": 24.0 * int(0.8 * n * case["deg"]) + 8 * n, "flops": 0}
    if kind == "recruit":
        rows, a = n + case["small"], case["nabd"]
        left = 0.01 * n + case["small"]
        return {"bytes": rows * (4 * a + 24.0), "flops": left * _genomes(n) * 10.0 * 2 * a}
    # three products of each layer per row, forward and two backward
    mac = NTNF * 256 + 256 * 128 + 128 * 64
    return {"bytes": n * (NTNF * 4 + 8) + 8.0 * case["pairs"],
            "flops": case["steps"] * 2.0 * case["batch"] * 6.0 * mac + 136.0 * n * (n - 1)}


# ------------------------------------------------------------------ exact --

# canonical tetranucleotides in column order, and the probability model's
# coefficients: powers of x (smaller log size), of y (larger) and of x * y
_TN = ("GGTAAGCCAAAAACATAGTCACGACATACGAAAAGTCAAACCAGGGACATTAGATCCCTCCTAAACTAAGGCGCAACCGCCGCCAAAC"
       "ACTCATCCGACCGAGAATAGATCACAGAAGTAATGAAAATTTAATATAAGTGAGCTCCACGGCCACCCGGGAGCGCATACCTGATAGA"
       "ATATGTCACTCCACAAACCTTAAAAACGCGAGAGGGATCGACGCTCAACTACCTCAGACAGGAACTTCGCCCCTGCTGCAGGCACACG"
       "GAGCAACTCATGAATTACAGAGATATAACATCGCCATCGACACACAACAAGGAGCAATGGATTCGTGAACCGGATAGCTACGTCCCCG"
       "AAGCCGTAGTACAGGAAATGCACCCAGCCGGCACACCCGGCCGACCCCTGAAAACAAGAGCCCACGGATACAACCAACGTGAACGTAA"
       "ATGCGTTATCCACAGGACTGAAAGAAGACAAGGCGAAACCACGGCCAACTTAAGACAGCGGAAAAATCATTGGCACCCTACGACCTAG"
       "AGAACGCACGCGAATA")
_B1 = ([46349.1624324381, -76092.3748553155, 53873.3933743949, -21263.6010657275, 5003.2646455284, -700.5825500292,
        54.037542743, -1.7713972342],
       [0, -639.918334183, -156.6547554844, 64.7719132839, -8.5014386744, 0.3968284526],
       [0, 474.0850141891, -23.966597785, 0.7800219061, -0.0138723693, 0.0001027543])
_C1 = ([-443565.465710869, 718862.10804858, -501588.206183097, 194712.394138513, -45088.7863182741, 6220.3310639927,
        -473.269785487, 15.3213264134],
       [0, 5114.1630934534, 784.4442123743, -377.9645994741, 50.5960513287, -2.3670776453],
       [0, -3282.8510348085, 164.0438603974, -5.2778800755, 0.0929379305, -0.0006826817])
_B2 = ([6770.9351457442, -5933.7589419767, 3279.7524685865, -967.2906583423, 159.8317289682, -14.0267151808,
        0.5108811613],
       [0, -2976.2879986855, 1602.7544794819, -462.0149190219, 74.4884405822, -6.3644917671, 0.2252455343],
       [0, 0, 0.965040193, -0.0546309127, 0.0012917084, -1.14383e-05])
_C2 = ([39406.5712626297, -77863.1741143294, 55360.1701572325, -21887.8400068324, 5158.3764225203, -724.0348081819,
        56.0522105105, -1.8470088417],
       [0, 9586.8761567725, -5825.2491611377, 1751.6803621934, -290.1765894829, 25.364646181, -0.9172073892],
       [0, 449.4660736502, -24.4141920625, 0.8465834103, -0.0158943762, 0.0001235384])


def _poly(c, v):
    r = torch.full_like(v, c[-1])
    for k in reversed(c[:-1]):
        r = r * v + k
    return r


def _prior(d, la, lb):
    """Pre-probabilities of pairs at distance d, log sizes la and lb."""
    x, y = torch.minimum(la, lb), torch.maximum(la, lb)

    def at(c):
        return _poly(c[0], x) + _poly(c[1], y) + _poly(c[2], x * y)

    ln9 = math.log(9.0)
    pre = -(at(_B1) + at(_C1) * d)
    pre2 = -(at(_B2) + at(_C2) * d)
    return torch.where(pre <= ln9, pre2.clamp(max=ln9), pre)


def _pre_block(ta, la, tb, lb):
    """Pre-probabilities of all pairs of two row sets, the distance's squares
    rounded to 32 bits and added in 64, as the model's definition has them."""
    d2 = torch.zeros(ta.shape[0], tb.shape[0], dtype=torch.float64, device=ta.device)
    for k in range(NTNF):
        e = ta[:, k, None] - tb[None, :, k]
        d2 += (e * e).double()
    return _prior(d2.sqrt_(), la[:, None], lb[None, :])


def _exact_graph(tnf, ls, cutoff, max_edges):
    """Scores in output order, zeros up to the buffer's size."""
    n = tnf.shape[0]
    L = math.log(1.0 / (1.0 - cutoff) - 1.0)
    out = []
    for i0 in range(0, n, 256):
        i1 = min(n, i0 + 256)
        pre = _pre_block(tnf[i0:i1], ls[i0:i1], tnf, ls)
        rows = torch.arange(i0, i1, device=tnf.device)
        pre[rows - i0, rows] = -math.inf
        sim = torch.where(pre > L, 1.0 - 1.0 / (1.0 + pre.exp()), 0.0)
        v, col = torch.sort(sim, dim=1, descending=True, stable=True)
        v, col = v[:, :max_edges], col[:, :max_edges]
        out.append(v[(v > 0) & (col > rows[:, None])])
    out = torch.cat(out)
    return torch.cat([out, out.new_zeros(n * min(max_edges, n - 1) - out.numel())])


def _exact_tnf(a):
    n = a["off"].numel()
    code = torch.full((256,), 4, dtype=torch.int64, device="cuda")
    for b, chars in enumerate((b"Aa", b"Cc", b"Gg", b"Tt")):
        for ch in chars:
            code[ch] = b
    num = {c: i for i, c in enumerate("ACGT")}
    column = torch.zeros(256, dtype=torch.int64, device="cuda")
    for k in range(NTNF):
        w = [num[c] for c in _TN[4 * k:4 * k + 4]]
        for q in (w, [3 - c for c in reversed(w)]):
            column[((q[0] * 4 + q[1]) * 4 + q[2]) * 4 + q[3]] = k
    ends = (a["off"] + a["len"]).cpu()
    res, i0 = [], 0
    while i0 < n:
        p0 = int(a["off"][i0])
        i1 = max(i0 + 1, int(torch.searchsorted(ends, p0 + (1 << 26))))
        p1 = int(ends[i1 - 1])
        x = a["buf"][p0:p1]
        pos = torch.arange(p0, p1, device="cuda")
        ctg = torch.searchsorted(a["off"][i0:i1].contiguous(), pos, right=True) - 1
        keep = (x != 10) & (pos < (a["off"][i0:i1] + a["len"][i0:i1])[ctg])
        b, ctg = code[x[keep].long()], ctg[keep]
        w = ((b[:-3] * 4 + b[1:-2]) * 4 + b[2:-1]) * 4 + b[3:]
        ok = (ctg[:-3] == ctg[3:]) & (torch.maximum(torch.maximum(b[:-3], b[1:-2]), torch.maximum(b[2:-1], b[3:])) < 4)
        c = torch.bincount(ctg[3:][ok] * NTNF + column[w[ok]], minlength=(i1 - i0) * NTNF).view(i1 - i0, NTNF)
        c = c.double()
        res.append(c / c.square().sum(1, keepdim=True).sqrt())
        i0 = i1
    return torch.cat(res)


def _exact_sscr(s):
    """Overlap of depth distributions per edge and sample, ranks and the
    weighted geometric mean, in 64 bits."""
    r1, r2, st = s["to"], s["fr"], s["st"]
    abd, var, ne = s["abd"], s["var"].clamp(min=1.0), s["st"].numel()
    raw = torch.zeros_like(st)
    nnz = torch.zeros_like(st)
    for i in range(abd.shape[1]):
        x, y = abd[r1, i], abd[r2, i]
        m1, m2 = x.clamp(min=1e-6), y.clamp(min=1e-6)
        v1, v2 = var[r1, i].sqrt() ** 2, var[r2, i].sqrt() ** 2
        t = (v1 * v2 * ((m1 - m2) ** 2 - 2 * (v1 - v2) * (v2 / v1).sqrt().log())).sqrt()
        near = (v2 - v1).abs() < 1e-4
        k1 = torch.where(near, (m1 + m2) / 2, (t - m1 * v2 + m2 * v1) / (v1 - v2))
        k2 = torch.where(near, (m1 + m2) / 2, (t + m1 * v2 - m2 * v1) / (v2 - v1))
        k1, k2 = torch.minimum(k1, k2), torch.maximum(k1, k2)

        def cdf(m, v, k):
            return 0.5 * torch.special.erfc(-(k - m) / (v.sqrt() * math.sqrt(2.0)))

        one = (cdf(m1, v1, k1) - cdf(m2, v2, k1)).abs()
        swap = v1 > v2
        ma, va = torch.where(swap, m2, m1), torch.where(swap, v2, v1)
        mb, vb = torch.where(swap, m1, m2), torch.where(swap, v1, v2)
        two = (cdf(ma, va, k2) - cdf(ma, va, k1) + cdf(mb, vb, k1) - cdf(mb, vb, k2)).abs()
        d = torch.where(m1 == m2, 0.0, torch.where(k1 == k2, one, two)).clamp(1e-6, 1 - 1e-6)
        use = (x > 1.0) | (y > 1.0)
        raw += torch.where(use, 1.0 - d, 0.0)
        nnz += use
    raw /= nnz
    distr = raw.sort().values
    w = 1.0 / (1.0 + nnz)
    rank = torch.searchsorted(st.sort().values, st)
    out = raw ** (1 - w) * distr[rank] ** w
    if abd.shape[1] >= 3:
        dev = abd - abd.mean(1, keepdim=True)
        norm = dev.square().sum(1).sqrt()
        cor = torch.zeros_like(st)
        for i in range(abd.shape[1]):
            cor += dev[r1, i] * dev[r2, i]
        cor /= norm[r1] * norm[r2]
        rank = torch.searchsorted(cor.sort().values, cor, right=True) - 1
        out = (out * distr[rank]).sqrt()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "labels", "recruit", "train"):
        return None  # whole numbers, or a long chain of rounded steps
    if kind == "graph" and case["n"] > 40000:
        return None
    s = prepare(case, seed)
    if kind == "count":
        return [None, _exact_tnf(s["a"])]
    if kind == "index":
        size = s["a"]["size"]
        ls = size[size >= 2500].clamp(max=500000).double().log10()
        return [None] * 6 + [torch.cat([ls, ls.new_zeros(size.numel() - ls.numel())]), None, None]
    if kind == "sample":
        pick = s["contigs"][:case["m"]]
        best = torch.full((case["m"],), -math.inf, dtype=torch.float64, device="cuda")
        for j0 in range(0, case["n"], 8192):
            j1 = min(case["n"], j0 + 8192)
            pre = _pre_block(s["tnf"][pick], s["log_size"][pick], s["tnf"][j0:j1], s["log_size"][j0:j1])
            pre[pick[:, None] == torch.arange(j0, j1, device="cuda")[None, :]] = -math.inf
            best = torch.maximum(best, pre.max(1).values)
        p = 1.0 - 1.0 / (1.0 + best.clamp(min=0.0).exp())
        return [torch.where(p >= case["floor"], p, 0.0)]
    if kind == "graph":
        return [None, None, None, _exact_graph(s["tnf"], s["log_size"], case["cutoff"], case["max_edges"])]
    if kind == "batch":
        return [None, None, None, torch.cat([_exact_graph(t, l, case["cutoff"], case["max_edges"])
                                             for t, l in s["sets"]])]
    return [_exact_sscr(s)]
