"""The work that is measured: graph builds through the package's public entry points.

A case is one FASTQ input (or a set of samples) and one way of building its graph.  `prepare`
makes the reads on the GPU from the seed alone, in the shapes of ``bruno_gb300.synth``'s
workloads (uniform genome, optional diverged repeat families, reads sampled uniformly with
random strand and uniform substitutions), and the context or pool that a program keeps between
builds; `run` is one build with its results taken out.  Tables and lists come in no particular
order from the library, so `run` puts them in the order of their k-mers.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import bruno_gb300 as bg

HEAD = 12            # "@r", nine digits, newline

SIZE_KEYS = ("n_reads", "n_reads_used", "n_instances", "n_k2", "n_nodes", "n_branch", "n_chain_nodes", "iterations",
             "n_cycle_nodes", "n_isolated", "n_ranked", "n_chains", "n_chain_chars")


def _case(name, form, k, genome, cov, len_lo, len_hi, sub, lower, *, host=False, repeats=0.0, n_frac=0.0,
          min_update=True, edge_filter=False, max_load=0.5, samples=1):
    return {"name": name, "form": form, "k": k, "genome": genome, "cov": cov, "len_lo": len_lo, "len_hi": len_hi,
            "sub": sub, "lower": lower, "host": host, "repeats": repeats, "n_frac": n_frac, "min_update": min_update,
            "edge_filter": edge_filter, "max_load": max_load, "samples": samples}


def listed():
    return [
        # one amplicon- or plasmid-sized request from host memory: the smallest call, all latency
        _case("tiny", "build", 31, 5_000, 20.0, 100, 100, 0.01, 2, host=True),
        # the benchmark's small workload (1 Mbp, 100k x 100 bp, 1%, -L 2) from host memory
        _case("small", "build", 31, 1_000_000, 10.0, 100, 100, 0.01, 2, host=True),
        # a bacterial genome at 30x from host memory, copied in pieces under the parsing
        _case("medium-host", "build", 31, 10_000_000, 30.0, 150, 150, 0.005, 3, host=True, repeats=0.02),
        # the benchmark's main workload: 50 Mbp + 2% repeats, 10M x 150 bp, FASTQ resident on the GPU
        _case("scale", "build", 31, 50_000_000, 30.0, 150, 150, 0.005, 3, repeats=0.02),
        # the large-k workload's mix (5% repeats, 150 bp, 30x, k = 63) at a tenth of its genome
        _case("large-k", "build", 63, 20_000_000, 30.0, 150, 150, 0.005, 3, repeats=0.05, max_load=0.7),
        # the reference driver's call sequence at an odd 128-bit k, reads trimmed to uneven lengths,
        # some with N, plain list ranking, the node table taken out
        _case("steps-ragged", "steps", 45, 1_234_567, 25.0, 61, 250, 0.01, 2, n_frac=0.02, min_update=False),
        # a build without thresholds (no -T): every erroneous k-mer becomes a node
        _case("unthresholded", "build", 31, 1_500_000, 12.0, 100, 151, 0.005, 0),
        # a short k on a small viral or bacterial genome at high coverage
        _case("short-k", "build", 21, 300_000, 200.0, 75, 100, 0.005, 5),
        # the blocked driver's (k+1)-mer edge filter
        _case("edge-filter", "build", 31, 2_000_000, 20.0, 100, 100, 0.01, 2, edge_filter=True),
        # the cleaning driver: dead ends and bubbles after the first compaction
        _case("clean", "clean", 31, 1_000_000, 25.0, 120, 150, 0.005, 1),
        # many samples of uneven size built in one fused pass, from host memory, chains out
        _case("batch", "batch", 31, 1_000_000, 40.0, 100, 250, 0.01, 2, host=True, samples=48),
        # a burst of requests through the served form (continuous batching)
        _case("served", "served", 31, 500_000, 30.0, 100, 200, 0.01, 2, host=True, samples=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["build", "build", "build", "build", "steps", "clean", "batch", "served"])
    sub = rng.choice([0.005, 0.01, 0.02])
    cov = round(rng.uniform(10.0, 60.0), 1)
    lo = rng.randint(75, 150)
    hi = rng.choice([lo, rng.randint(lo, 250)])
    lower = rng.choice([2, 3])
    if form in ("batch", "served"):
        return _case(form, form, 31, _log(rng, 20_000, 800_000), cov, 100, 250, sub, lower, host=True,
                     samples=rng.randint(3, 24))
    k = rng.choice([21, 25, 27, 29, 31, 31, 31, 31, 33, 45, 55, 63])
    genome = _log(rng, 5_000, 12_000_000 if form == "build" else 1_500_000)
    if genome * cov > 240_000_000:
        cov = 20.0
    ragged = hi > lo and genome * cov < 60_000_000
    if form == "build":
        opt = rng.choice(["", "", "", "edge", "none"]) if genome < 2_000_000 else ""
        return _case("build", "build", k, genome, cov, max(lo, k + 12), max(hi if ragged else lo, k + 12), sub,
                     0 if opt == "none" else lower, host=rng.random() < 0.4, repeats=rng.choice([0.0, 0.02, 0.05]),
                     n_frac=rng.choice([0.0, 0.01]), edge_filter=opt == "edge",
                     max_load=0.7 if k > 31 else 0.5)
    return _case(form, form, k, genome, cov, max(lo, k + 12), max(hi if ragged else lo, k + 12), sub, lower,
                 n_frac=rng.choice([0.0, 0.01]), min_update=rng.random() < 0.7)


# ------------------------------------------------------------------------------ inputs
def _genome(gen, n, repeats):
    """uniform bases (0..3); `repeats` of it are segments copied elsewhere with 1% divergence"""
    g = torch.randint(0, 4, (n,), generator=gen, device="cuda", dtype=torch.uint8)
    left = int(n * repeats)
    if left < 1000:
        return g
    r = torch.randint(0, 1 << 30, (4096,), generator=gen, device="cuda").tolist()
    at = 0
    while left > 1000 and at + 20 < len(r):
        length = min(1000 + r[at] % 9000, left, n // 4)
        copies = 2 + r[at + 1] % 7
        src = r[at + 2] % (n - length)
        at += 3
        seg = g[src:src + length].clone()
        for _ in range(copies):
            if left <= 0:
                break
            dst = r[at] % (n - length)
            at += 1
            mut = torch.rand(length, generator=gen, device="cuda") < 0.01
            sub = torch.randint(1, 4, (length,), generator=gen, device="cuda", dtype=torch.uint8)
            g[dst:dst + length] = torch.where(mut, (seg + sub) & 3, seg)
            left -= length
    return g


def _reads(gen, g, lens, first, sub, n_frac, fixed):
    """FASTQ bytes of len(lens) reads, numbered from `first`"""
    n, G = lens.numel(), g.numel()
    dev = g.device
    ascii4 = torch.tensor([65, 67, 71, 84], dtype=torch.uint8, device=dev)
    start = (torch.rand(n, generator=gen, device=dev, dtype=torch.float64) * (G - lens + 1)).long()
    rc = torch.rand(n, generator=gen, device=dev) < 0.5
    has_n = torch.rand(n, generator=gen, device=dev) < n_frac
    ids = torch.arange(first, first + n, device=dev)
    digits = torch.stack([(ids // 10 ** (8 - j)) % 10 for j in range(9)], 1).to(torch.uint8) + 48
    if fixed:
        L = fixed
        out = torch.empty((n, HEAD + 2 * L + 4), dtype=torch.uint8, device=dev)
        j = torch.arange(L, device=dev)
        pos = start[:, None] + torch.where(rc[:, None], L - 1 - j, j)
        b = g[pos]
        del pos
        b = torch.where(rc[:, None], 3 - b, b)
        mut = torch.rand((n, L), generator=gen, device=dev) < sub
        b = torch.where(mut, (b + torch.randint(1, 4, (n, L), generator=gen, device=dev, dtype=torch.uint8)) & 3, b)
        seq = ascii4[b.long()]
        if n_frac:
            seq[:, L // 2] = torch.where(has_n, torch.full_like(seq[:, 0], 78), seq[:, L // 2])
        out[:, 0], out[:, 1] = 64, 114
        out[:, 2:11] = digits
        out[:, 11] = 10
        out[:, HEAD:HEAD + L] = seq
        out[:, HEAD + L], out[:, HEAD + L + 1], out[:, HEAD + L + 2] = 10, 43, 10
        out[:, HEAD + L + 3:HEAD + 2 * L + 3] = 73
        out[:, HEAD + 2 * L + 3] = 10
        return out.reshape(-1)
    rec = HEAD + 2 * lens + 4
    off = torch.cumsum(rec, 0) - rec
    total = int(rec.sum())
    r = torch.repeat_interleave(torch.arange(n, device=dev), rec, output_size=total)
    p = torch.arange(total, device=dev) - off[r]
    L = lens[r]
    out = torch.full((total,), 73, dtype=torch.uint8, device=dev)
    q = p - HEAD
    in_seq = (q >= 0) & (q < L)
    gp = (start[r] + torch.where(rc[r], L - 1 - q, q)).clamp_(0, G - 1)
    b = torch.where(rc[r], 3 - g[gp], g[gp])
    mut = torch.rand(total, generator=gen, device=dev) < sub
    b = torch.where(mut, (b + torch.randint(1, 4, (total,), generator=gen, device=dev, dtype=torch.uint8)) & 3, b)
    seq = ascii4[b.long()]
    seq[has_n[r] & (q == L // 2)] = 78
    out = torch.where(in_seq, seq, out)
    out[(q == -1) | (q == L) | (q == L + 2) | (p == rec[r] - 1)] = 10
    out[q == L + 1] = 43
    head = p < HEAD - 1
    hd = torch.cat([torch.tensor([[64, 114]], dtype=torch.uint8, device=dev).expand(n, 2), digits], 1)
    out[head] = hd[r[head], p[head]]
    return out


def _fastq(seed, genome, cov, lo, hi, sub, repeats, n_frac):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = min(lo, genome), min(hi, genome)
    g = _genome(gen, genome, repeats)
    n = max(1, int(round(genome * cov / ((lo + hi) / 2))))
    step = 1_000_000 if lo == hi else 200_000
    parts = []
    for a in range(0, n, step):
        m = min(step, n - a)
        lens = torch.full((m,), lo, device="cuda", dtype=torch.long) if lo == hi else \
            torch.randint(lo, hi + 1, (m,), generator=gen, device="cuda")
        parts.append(_reads(gen, g, lens, a, sub, n_frac, lo if lo == hi else 0))
    return torch.cat(parts) if len(parts) > 1 else parts[0]


def _to_host(t):
    """page-locked host copy, as a program that reads files into reusable buffers holds it"""
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)
    h.copy_(t)
    return h


def _sample_shapes(case, seed):
    """samples of uneven size: genome log-uniform from 5 kbp to the case's, their own coverage and
    read length; the seed changes the reads, not the sizes"""
    rng = np.random.default_rng(case["samples"])
    out = []
    for i in range(case["samples"]):
        g = int(round(np.exp(rng.uniform(np.log(5_000), np.log(case["genome"])))))
        cov = float(rng.uniform(0.5, 1.5)) * case["cov"]
        out.append((g, cov, int(rng.integers(case["len_lo"], case["len_hi"] + 1)), seed * 4096 + i))
    return out


def prepare(case, seed):
    k, lower = case["k"], case["lower"]
    cfg = bg.GraphConfig(k=k, thresholding=lower > 0, thresh=bg.thresholds([lower] if lower else []),
                         min_update=case["min_update"], edge_filter=case["edge_filter"], max_load=case["max_load"])
    st = {"case": case, "form": case["form"]}
    if case["form"] in ("batch", "served"):
        parts = [_fastq(s, g, cov, L, L, case["sub"], 0.0, 0.0) for g, cov, L, s in _sample_shapes(case, seed)]
        host = _to_host(torch.cat(parts))
        cuts = np.concatenate([[0], np.cumsum([p.numel() for p in parts])])
        st["keep"] = host
        a = host.numpy()
        st["inputs"] = [a[cuts[i]:cuts[i + 1]] for i in range(len(parts))]
    else:
        fq = _fastq(seed, case["genome"], case["cov"], case["len_lo"], case["len_hi"], case["sub"], case["repeats"],
                    case["n_frac"])
        st["keep"] = _to_host(fq) if case["host"] else fq
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    if case["form"] == "served":
        st["pool"] = bg.Pool(cfg, batched=True, max_samples=64, mem_budget=16 << 30)
    else:
        st["stream"] = torch.cuda.Stream()
        st["graph"] = bg.Graph(cfg)
        st["graph"].set_stream(st["stream"].cuda_stream)
    return st


def _room(case):
    """most chains, chain characters and nodes the case's graphs have: the genome, and per error
    that `lower` reads or more share k nodes and up to four chain ends"""
    genome, k = case["genome"], case["k"]
    if case["form"] in ("batch", "served"):
        genome *= case["samples"]
    lam, need = 1.5 * case["cov"] * case["sub"] / 3, max(1, case["lower"])
    kept = 1 - sum(math.exp(-lam) * lam ** i / math.factorial(i) for i in range(need))
    err = 3 * genome * kept * 1.5
    return {"chains": int(4 * err + genome / 20) + 4096, "chars": int(4 * k * err + 3 * genome) + 65536,
            "nodes": int(k * err + 2 * genome) + 65536}


def _padded(t, n):
    if t.shape[0] > n:
        raise RuntimeError("more results than the case has room for: %d > %d" % (t.shape[0], n))
    out = torch.zeros((n,) + tuple(t.shape[1:]), dtype=t.dtype, device=t.device)
    out[:t.shape[0]] = t
    return out


# ------------------------------------------------------------------------------ one pass
class _View:
    """a read-only device array of the library's, for torch.as_tensor"""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _device(ptr, shape, typestr, dtype):
    if math.prod(shape) == 0:
        return torch.empty(shape, dtype=dtype, device="cuda")
    return torch.as_tensor(_View(ptr, shape, typestr), device="cuda")


def _order(keys):
    """the order of k-mers (n, words), the last word the most significant"""
    o = torch.sort(keys[:, 0]).indices
    if keys.shape[1] > 1:
        o = o[torch.sort(keys[o, 1], stable=True).indices]
    return o


def _chains(room, reps, offs, chars, group=None):
    """chains in the order of their representatives (within `group`, if given), as whole arrays"""
    o = _order(reps)
    if group is not None:
        o = o[torch.sort(group[o], stable=True).indices]
    lens = offs[1:] - offs[:-1]
    new = torch.cumsum(lens[o], 0)
    at = torch.repeat_interleave(offs[:-1][o] - (new - lens[o]), lens[o], output_size=chars.numel())
    at += torch.arange(chars.numel(), device=at.device)
    return {"reps": _padded(reps[o], room["chains"]), "ends": _padded(new, room["chains"]),
            "chars": _padded(chars[at], room["chars"])}


def _dev(a):
    return torch.from_numpy(a.view(np.int64) if a.dtype == np.uint64 else a).cuda(non_blocking=True)


def _sizes(s):
    return np.array([s[n] for n in SIZE_KEYS] + list(s.get("filter_flag_hist", [])), dtype=np.int64)


def _nodes(g, room):
    keys, counts, flags = g.nodes()
    keys = _dev(keys)
    o, n = _order(keys), room["nodes"]
    return {"keys": _padded(keys[o], n), "counts": _padded(_dev(counts.view(np.int16))[o], n),
            "flags": _padded(_dev(flags)[o], n)}


def _out(g, case):
    out, room = {"sizes": _sizes(g.sizes())}, _room(case)
    if case["host"]:     # a program with host buffers takes host buffers back
        reps, offs, chars = g.chains()
        out["chains"] = _chains(room, _dev(reps), _dev(offs), _dev(chars))
        return out
    d = g.device_results()
    w, nc, nr = d["words"], d["n_chains"], d["n_ranked"]
    out["chains"] = _chains(room, _device(d["chain_reps"], (nc, w), "<i8", torch.int64),
                            _device(d["chain_offsets"], (nc + 1,), "<i8", torch.int64),
                            _device(d["chain_chars"], (d["n_chain_chars"],), "|u1", torch.uint8))
    if case["genome"] <= 2_000_000:
        K = _device(d["ranked_K"], (nr, w), "<i8", torch.int64)
        o, n = _order(K), room["nodes"]
        out["ranked"] = {"K": _padded(K[o], n), "rep": _padded(_device(d["ranked_rep"], (nr, w), "<i8", torch.int64)[o], n),
                         "dist": _padded(_device(d["ranked_dist"], (nr,), "<i4", torch.int32)[o], n)}
    return out


def _joined(room, parts):
    """many samples' chains (reps, offsets, chars) as one set of arrays, sample after sample"""
    lens = np.array([len(c) for _, _, c in parts], dtype=np.int64)
    base = np.cumsum(lens) - lens
    offs = np.concatenate([o[:-1].astype(np.int64) + b for (_, o, _), b in zip(parts, base)] + [[int(lens.sum())]])
    group = np.repeat(np.arange(len(parts)), [len(r) for r, _, _ in parts])
    return _chains(room, _dev(np.concatenate([r for r, _, _ in parts])), _dev(offs),
                   _dev(np.concatenate([c for _, _, c in parts])), _dev(group))


def run(st):
    case, form = st["case"], st["form"]
    if form == "served":
        pool = st["pool"]
        got = [pool.wait(t) for t in [pool.submit(a) for a in st["inputs"]]]
        if any(r["status"] for r in got):
            raise RuntimeError("a request failed: %s" % [r["status"] for r in got])
        return {"sizes": np.stack([_sizes(r["sizes"]) for r in got]), "chains": _joined(_room(case), [r["chains"] for r in got])}
    g, data = st["graph"], st["keep"]
    with torch.cuda.stream(st["stream"]):
        if form == "batch":
            g.build_samples(st["inputs"])
            n = len(st["inputs"])
            return {"sizes": np.stack([_sizes(g.sample_sizes(i)) for i in range(n)]),
                    "chains": _joined(_room(case), g.batch_chains())}
        if form == "steps":      # the reference driver's sequence, its node table taken out before ranking
            g.reset()
            g.load_fastq(data.data_ptr(), data.numel(), is_device=True)
            g.compute_biedge_freqencies()
            g.local_insert_by_freqencies()
            nodes = _nodes(g, _room(case))
            g.extract_chains()
            g.list_rank_min_update() if case["min_update"] else g.list_rank()
            g.to_compressed_chains()
            return dict(_out(g, case), nodes=nodes)
        if case["host"]:
            g.build_and_compact(data.numpy())
        else:
            g.build_and_compact(data.data_ptr(), data.numel(), is_device=True)
        if form == "clean":
            stats = g.clean_deadend_and_bubbles_naive()
            return dict(_out(g, case), clean=np.array([stats[n] for n in ("rounds", "deadends", "bubbles", "edges")]))
        return _out(g, case)


def work(case):
    """the FASTQ read once, the chains (and what else comes out) written once"""
    mean = (case["len_lo"] + case["len_hi"]) / 2
    # samples are log-uniform from 5 kbp to `genome`
    genome = case["genome"] if case["form"] not in ("batch", "served") else \
        case["samples"] * (case["genome"] - 5_000) / max(1e-9, math.log(case["genome"] / 5_000))
    reads = genome * case["cov"] / mean
    out = genome * (1 + (20 * (1 + (case["k"] > 31)) if case["genome"] <= 2_000_000 and not case["host"] else 0))
    return {"bytes": reads * (HEAD + 2 * mean + 4) + out, "flops": 0}


def exact(case, seed):
    """every output is a whole number or a byte: there is nothing to be rounded"""
    return None
