"""Super-k-mer builds where an input outgrows what its plan foresaw, against the oracle and against the
plain build: more records than their room, cycles within one block of chain nodes, pointers that disagree,
partitions with more k-mers or records than a block counts, reads of k + 1 bases under the (k+1)-mer filter."""
import subprocess
import sys

import numpy as np
import pytest

import bruno_gb300 as bg
from helpers import assert_same, chain_set, compress_ranked, sort_nodes, sort_ranked
from oracle import oracle
from test_gpu_batch import batch, plain, same_as_plain
from test_gpu_parity import compare, gpu_run
from test_gpu_superkmers import low_mmer

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)
SIZES = ("n_reads", "n_reads_used", "n_instances", "n_k2", "n_nodes", "n_branch", "n_chain_nodes", "iterations",
         "n_cycle_nodes", "n_isolated", "n_ranked", "n_chains", "n_chain_chars")


def rand_reads(rng, genome, n, length, err=0.0):
    """n x length base codes of reads of either strand"""
    at = rng.integers(0, len(genome) - length + 1, n)
    c = genome[at[:, None] + np.arange(length)]
    if err:
        c = np.where(rng.random(c.shape) < err, (c + rng.integers(1, 4, c.shape)) & 3, c)
    flip = rng.random(n) < 0.5
    c[flip] = 3 - c[flip][:, ::-1]
    return c


def fastq(codes, qual=None):
    """records of one read length, with `qual` quality characters (the read's length by default)"""
    n, length = codes.shape
    q = length if qual is None else qual
    out = np.empty((n, 7 + length + q), dtype=np.uint8)
    out[:, :3] = np.frombuffer(b"@r\n", dtype=np.uint8)
    out[:, 3:3 + length] = ACGT[codes]
    out[:, 3 + length:6 + length] = np.frombuffer(b"\n+\n", dtype=np.uint8)
    out[:, 6 + length:6 + length + q] = ord("I")
    out[:, 6 + length + q] = 10
    return out.tobytes()


def check(data, k, thr, thresholding=True, superkmers=True, **cfg):
    """a one-call build (by super-k-mers, unless said) against the oracle; returns its sizes"""
    ref = oracle.run(data, k=k, thresholding=thresholding, thresh=thr, min_update=True, threads=16,
                     edge_filter=cfg.get("edge_filter", False))
    with bg.Graph(k=k, thresholding=thresholding, thresh=thr, min_update=True, **cfg) as g:
        g.build_and_compact(data)
        assert (g.counting_path()[0] == "super_kmers") == superkmers
        s = g.sizes()
        for n in SIZES:
            if n in ref:
                assert s[n] == ref[n], (n, s[n], ref[n])
        assert_same(sort_nodes(*g.nodes()), ref["nodes"], "graph nodes")
        assert_same(sort_ranked(*g.ranked()), ref["ranked"], "listranked chain nodes")
        assert chain_set(*g.chains()) == chain_set(*ref["chains"])
        return s


# ------------------------------------------------------------------ more records than their room
@pytest.mark.parametrize("k,chunk", [(21, 0), (21, 16 << 20), (33, 0)])
def test_quality_lines_of_one_character(k, chunk):
    """a quality line need not be as long as its sequence: nearly every byte is then a k-mer position,
    and the records outgrow the room that half the bytes would need (24000 reads of 1 kb, k = 21: 5.8M
    records, places for 4.7M; k = 33: 2.3M, places for 2.1M); at once and in pieces of a host copy"""
    rng = np.random.default_rng(k)
    data = fastq(rand_reads(rng, rng.integers(0, 4, 300_000), 24_000, 1000, 0.002), qual=1)
    check(data, k, bg.thresholds([2]), h2d_chunk=chunk)


@pytest.mark.parametrize("chunk", [0, 16 << 20])
def test_quality_lines_of_one_character_in_a_batch(chunk):
    rng = np.random.default_rng(chunk + 1)
    samples = [fastq(rand_reads(rng, rng.integers(0, 4, 150_000), n, 1000, 0.002), qual=1)
               for n in (9_000, 300, 9_000, 9_000)]
    cfg = dict(k=21, thresholding=True, thresh=bg.thresholds([2]), min_update=True)
    got, _ = batch(samples, h2d_chunk=chunk, **cfg)
    for i, data in enumerate(samples):
        same_as_plain(got[i], plain(data, **cfg), f"sample {i}")


# ------------------------------------------------------------------ segments of chain nodes
@pytest.mark.parametrize("k", [31, 63])
def test_circular_genomes_within_one_block(k):
    """cycles whose nodes all lie in one block of the segment search (2048 nodes), around its edge, and
    beside a linear genome"""
    rng = np.random.default_rng(k)
    for n in (k + 3, 150, 256, 777, 1024, 2047, 2048, 2049):
        g = rng.integers(0, 4, n)
        at = np.concatenate([np.arange(0, n, 3), rng.integers(0, n, 100)])
        reads = g[(at[:, None] + np.arange(100)) % n]
        reads[::2] = 3 - reads[::2][:, ::-1]
        data = fastq(reads)
        s = check(data, k, bg.thresholds([1]))
        assert s["n_cycle_nodes"] == n and s["n_ranked"] == 0
        line = rng.integers(0, 4, 1500)
        check(data + fastq(rand_reads(rng, line, 300, 100)), k, bg.thresholds([1]))


@pytest.mark.parametrize("k", [21, 31, 45])
def test_small_inconsistent_chain_maps(k):
    """separate k and k+2 bounds on graphs of a few blocks: pointers that disagree inside a block and
    between blocks; the compaction must be that of the listranked nodes, everything before it the oracle's"""
    thr = [2, 65536, 2, 65536, 2, 65536]
    for seed in range(12):
        rng = np.random.default_rng(100 * k + seed)
        genome = rng.integers(0, 4, int(rng.integers(200, 6000)))
        data = fastq(rand_reads(rng, genome, 6 * len(genome) // 100, 100, 0.01))
        ref = oracle.run(data, k=k, thresh=thr, min_update=True)
        with bg.Graph(k=k, thresh=thr, min_update=True) as g:
            g.build_and_compact(data)
            assert g.sizes()["n_chain_nodes"] == ref["n_chain_nodes"]
            assert_same(sort_nodes(*g.nodes()), ref["nodes"], "graph nodes")
            assert chain_set(*g.chains()) == compress_ranked(*g.ranked(), k)


# ------------------------------------------------------------------ crowded partitions
ADAPTER = np.array(["ACGT".index(c) for c in "AGATCGGAAGAGCACACGTCTGAACTCCAGTCA"] + [0] * 200)


def tailed(rng, codes, n, tail):
    """n of the reads end in `tail`, from a place of their own on"""
    c = codes.copy()
    length = c.shape[1]
    for i in rng.choice(len(c), n, replace=False):
        p = int(rng.integers(8, length - 20))
        c[i, p:] = tail[:length - p]
    return c


def crowded_reads(kind, seed, n=24_000, genome=120_000):
    """reads of 100 bases whose k-mers crowd one minimizer or a few: the places where an adapter or a run
    of one base begins (more k-mers than a block's slots), whole reads of one base (more records than a
    block counts), a diverged satellite"""
    rng = np.random.default_rng(seed)
    g = rng.integers(0, 4, genome)
    if kind == "satellite":
        unit = rng.integers(0, 4, 171)
        for p in range(0, genome - 2000, 4000):
            t = np.resize(unit, 2000)
            g[p:p + 2000] = np.where(rng.random(2000) < 0.1, (t + rng.integers(1, 4, 2000)) & 3, t)
    c = rand_reads(rng, g, n, 100, 0.003)
    if kind == "adapter":
        c = tailed(rng, c, n // 3, ADAPTER)
    elif kind == "poly-A":
        c = tailed(rng, c, n // 3, np.zeros(200, dtype=int))
    elif kind == "one base":
        c[rng.random(n) < 0.4] = 3
    return c


@pytest.mark.parametrize("thr", [[2], []])
@pytest.mark.parametrize("kind", ["adapter", "poly-A", "one base", "satellite"])
@pytest.mark.parametrize("k", [21, 31, 45, 63])
def test_crowded_partitions(k, kind, thr):
    """one call, and the step calls with every count copied out (k = 21 keeps every k-mer by k-mer records)"""
    data = fastq(crowded_reads(kind, k))
    check(data, k, bg.thresholds(thr), thresholding=bool(thr), superkmers=bool(thr) or k > 21)
    ref = oracle.run(data, k=k, thresholding=bool(thr), thresh=bg.thresholds(thr), min_update=True, keep_k2=True,
                     keep_filtered=True, threads=16)
    compare(gpu_run(data, k, bool(thr), bg.thresholds(thr), True), ref)


@pytest.mark.parametrize("kind", ["adapter", "one base"])
@pytest.mark.parametrize("k", [21, 30, 31, 63])
def test_crowded_partitions_edge_filter(k, kind):
    check(fastq(crowded_reads(kind, 7 * k)), k, bg.thresholds([3]), edge_filter=True)


@pytest.mark.parametrize("chunk", [0, 1 << 20])
def test_crowded_samples_of_a_batch(chunk):
    """samples that crowd a partition among samples that do not, in one copy and in groups"""
    rng = np.random.default_rng(11)
    samples = [fastq(rand_reads(rng, rng.integers(0, 4, 20_000), 3_000, 100, 0.003)) for _ in range(6)]
    for at, kind in ((1, "adapter"), (4, "one base"), (6, "poly-A")):
        samples.insert(at, fastq(crowded_reads(kind, at)))
    cfg = dict(k=31, thresholding=True, thresh=bg.thresholds([2]), min_update=True)
    got, _ = batch(samples, h2d_chunk=chunk, **cfg)
    for i, data in enumerate(samples):
        same_as_plain(got[i], plain(data, **cfg), f"sample {i}")


def test_crowded_partitions_cleaned():
    """cleaning looks nodes up, erases them and lists them again: in a table with crowded partitions too"""
    data = fastq(crowded_reads("adapter", 3))
    thr = bg.thresholds([1])
    ref = oracle.run(data, k=31, thresh=thr, min_update=True, threads=16, clean=True)
    with bg.Graph(k=31, thresh=thr, min_update=True) as g:
        g.build_and_compact(data)
        stats = g.clean_deadend_and_bubbles_naive()
        for n in ("rounds", "deadends", "bubbles", "edges"):
            assert stats[n] == ref["clean_stats"][n], n
        assert_same(sort_nodes(*g.nodes()), ref["clean"]["nodes"], "cleaned nodes")
        assert chain_set(*g.chains()) == chain_set(*ref["clean"]["chains"])


@pytest.mark.parametrize("k", [31, 45])
def test_a_count_past_what_a_block_may_hold(k):
    """one biedge of one k-mer counted more than 2^25 times (300 bases a read, all alike, beside a
    genome's reads): capped where only the filter reads it, exact where the counts are copied out, by the side
    table of counts past an entry's own"""
    n = (1 << 25) // (300 - k - 1) + 2000
    rng = np.random.default_rng(k)
    data = fastq(np.zeros((n, 300), dtype=np.int8)) + fastq(rand_reads(rng, rng.integers(0, 4, 30_000), 6_000, 100, 0.003))
    check(data, k, bg.thresholds([2]))
    ref = oracle.run(data, k=k, thresh=bg.thresholds([2]), min_update=True, keep_k2=True, keep_filtered=True, threads=16)
    assert int(ref["k2"][2].max()) > 1 << 25
    compare(gpu_run(data, k, True, bg.thresholds([2]), True), ref)


ESTIMATE = r"""
import numpy as np, torch
import bruno_gb300 as bg
c = np.load("{reads}")
name = b"@" + b"r" * 10000
data = b"".join(name + b"\n" + r.tobytes() + b"\n+\n" + b"I" * len(r) + b"\n" for r in c)
torch.zeros(1, device="cuda")
before = torch.cuda.mem_get_info()[0]
with bg.Graph(k=31, thresh=bg.thresholds([2]), min_update=True) as g:
    g.build_and_compact(data)
    print(g.sizes()["n_instances"], (before - torch.cuda.mem_get_info()[0]) >> 20)
"""


def test_estimate_with_a_crowded_minimizer_in_its_sample(tmp_path):
    """the distinct estimate samples one minimizer in 32 of a 61 MB input; with 6000 places on one that is
    in the sample it comes to 3.8M, but the table is planned for no more than the 0.63M k-mers there are
    (the build then holds some 200 MB, 210 MB less than with slots for the estimate)"""
    rng = np.random.default_rng(2)
    pack = lambda v: int("".join(f"{int(x):02b}" for x in v), 2)
    while True:   # an M-mer of a small order whose bin bits end in five zeros (kmer.cuh mz_order, mz_mix)
        fwd = np.array(["ACGT".index(c) for c in low_mmer(int(rng.integers(1 << 30)))])
        h = ((min(pack(fwd), pack(3 - fwd[::-1])) ^ 0x2C9277B5) * 0x9E3779B1 & 0xFFFFFFFE) >> 1
        h = h * 0xC2B2AE35 & 0xFFFFFFFF
        h = (h ^ (h >> 15)) * 0x27D4EB2F & 0xFFFFFFFF
        if (h ^ (h >> 16)) & 31 == 0:
            break
    c = rng.integers(0, 4, (6000, 135))
    c[:, 60:75] = fwd
    np.save(tmp_path / "reads.npy", ACGT[c])
    r = subprocess.run([sys.executable, "-c", ESTIMATE.format(reads=tmp_path / "reads.npy")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    instances, held = (int(x) for x in r.stdout.split())
    assert instances == 6000 * 105 and held < 300, held


# ------------------------------------------------------------------ reads of k + 1 bases under the (k+1)-mer filter
def trimmed(codes, lens):
    return b"".join(b"@r\n" + ACGT[c[:n]].tobytes() + b"\n+\n" + b"I" * int(n) + b"\n" for c, n in zip(codes, lens))


@pytest.mark.parametrize("share", [0.002, 0.3, 1.0])
@pytest.mark.parametrize("k", [19, 22, 31, 32, 45, 63])
def test_edge_filter_with_reads_of_k_plus_1_bases(k, share):
    """reads cut to k + 1 bases beside longer ones, few, many or all: their (k+1)-mers decide which edges
    the others keep; homopolymers and palindromes among them"""
    rng = np.random.default_rng(k)
    genome = rng.integers(0, 4, 3000)
    half = rng.integers(0, 4, (k + 1) // 2)
    genome[500:500 + 2 * len(half)] = np.concatenate([half, 3 - half[::-1]])
    genome[900:960] = 0
    c = rand_reads(rng, genome, 4000, 100, 0.01)
    lens = np.where(rng.random(4000) < share, k + 1, rng.integers(k, 101, 4000))
    data = trimmed(c, lens)
    for lo, hi in ((2, 65536), (4, 65536), (2, 12)):
        check(data, k, np.array([0, 65536, lo, hi, 0, 65536], dtype=np.uint64), edge_filter=True)


def test_edge_filter_with_crowded_reads_of_k_plus_1_bases():
    rng = np.random.default_rng(4)
    c = crowded_reads("adapter", 5)
    data = trimmed(c, np.where(rng.random(len(c)) < 0.2, 32, 100)) + trimmed(np.zeros((40_000, 32), dtype=int), [32] * 40_000)
    check(data, 31, bg.thresholds([3]), edge_filter=True)


# ------------------------------------------------------------------ more than 2^32 k-mers
def test_more_than_2_32_kmers():
    """a 30x build of 5 Mbp whose input comes 29 times over: 4.35G k-mers, the graph of the input once with 29
    times the counts, by super-k-mers"""
    import torch
    rng = np.random.default_rng(8)
    one = fastq(rand_reads(rng, rng.integers(0, 4, 5_000_000), 1_250_000, 150, 0.005))
    n = 29

    def build(data, size, lower):
        with bg.Graph(k=31, thresh=bg.thresholds([lower]), min_update=True) as g:
            g.build_and_compact(data.data_ptr(), size, is_device=True)
            assert g.counting_path()[0] == "super_kmers"
            return g.sizes(), sort_nodes(*g.nodes()), chain_set(*g.chains())

    a = torch.from_numpy(np.frombuffer(one, dtype=np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    s1, nodes1, chains1 = build(a, a.numel(), 3)
    b = a.repeat(n)
    del a
    torch.cuda.synchronize()   # the library's stream does not wait for torch's
    s, nodes, chains = build(b, b.numel(), 3 * n)
    assert s["n_instances"] == n * s1["n_instances"] > 1 << 32
    for key in ("n_k2", "n_nodes", "n_branch", "n_chain_nodes", "n_chains"):
        assert s[key] == s1[key], key
    assert_same((nodes[0], nodes[2]), (nodes1[0], nodes1[2]), "nodes")
    assert np.array_equal(nodes[1], np.minimum(65535, n * nodes1[1].astype(np.int64)).astype(nodes[1].dtype))
    assert chains == chains1


# ------------------------------------------------------------------ the estimate's error
@pytest.mark.parametrize("thr", [[2], []])
def test_estimates_within_the_table(thr):
    """builds that keep every k-mer are counted once: an estimate some percent low, as a sample of minimizers
    often is, still leaves the table room (a second attempt shows as launches; some of these 32 inputs needed
    one)"""
    launches = []
    for seed in range(32):
        rng = np.random.default_rng(1000 + seed)
        data = fastq(rand_reads(rng, rng.integers(0, 4, 150_000), 60_000, 100, 0.01))
        with bg.Graph(k=31, thresholding=bool(thr), thresh=bg.thresholds(thr), min_update=True) as g:
            g.load_fastq(data)
            g.compute_biedge_freqencies()
            assert g.counting_path()[0] == "super_kmers"
            launches.append(g.sizes()["launches"])
    assert len(set(launches)) == 1, launches


def test_every_partition_crowded_by_records():
    """a genome of 2200 bases at 60000x: more than half of the partitions hold more records than a block counts,
    which says nothing about the estimate, so that the plan stays (a further attempt shows as launches)"""
    rng = np.random.default_rng(6)
    data = fastq(rand_reads(rng, rng.integers(0, 4, 2200), 1_300_000, 100))
    s = check(data, 31, bg.thresholds([2]))
    assert s["n_nodes"] <= 2170 and s["table_partitions"] == 256 and s["launches"] < 48, s["launches"]


@pytest.mark.parametrize("k", [31, 45])
def test_crowded_partitions_with_wide_kmers_and_other_thresholds(k):
    """a k-mer between every pair of bases in a crowded partition (more biedges than a slot holds), and the
    filter with other thresholds than the count's, which reads every slot"""
    rng = np.random.default_rng(k)
    c = crowded_reads("poly-A", k)
    wide = np.array([np.concatenate([rng.integers(0, 4, 50 - k // 2), [a], np.zeros(k, dtype=int), [b],
                                     rng.integers(0, 4, 100)])[:100] for a in range(4) for b in range(4)] * 3)
    data = fastq(np.concatenate([c, wide]))
    check(data, k, bg.thresholds([2]))
    for thr in ([3], [1], [1, 2, 3]):
        t = bg.thresholds(thr)
        ref = oracle.run(data, k=k, thresh=t, min_update=True, threads=16)
        with bg.Graph(k=k, thresh=bg.thresholds([2]), min_update=True) as g:
            g.load_fastq(data)
            g.compute_biedge_freqencies()
            assert g.counting_path()[0] == "super_kmers"
            g.local_insert_by_freqencies(t)
            assert g.sizes()["n_nodes"] == ref["n_nodes"] and g.sizes()["filter_flag_hist"] == ref["filter_flag_hist"]
            assert_same(sort_nodes(*g.nodes()), ref["nodes"], f"graph nodes, {thr}")
