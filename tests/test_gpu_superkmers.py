"""Counting by super-k-mers at the sizes where its kernels can go wrong, against the oracle: reads
around the 16-base words and the 512-base tiles of the extraction, every window-block size (k - 15
from 4, from 8, from 16), homopolymers and short repeats (one minimizer over a whole read), N and
lowercase bases, and partitions with more k-mers than their block's shared-memory slots."""
import numpy as np
import pytest

import bruno_gb300 as bg
from helpers import assert_same, chain_set, sort_nodes, sort_ranked
from oracle import oracle
from test_gpu_batch import batch, plain, same_as_plain
from test_gpu_parity import compare, compare_one_call, gpu_run, one_call_run

pytestmark = pytest.mark.gpu

M = 15


def fastq(reads):
    return "".join(f"@r{i}\n{s}\n+\n{'I' * len(s)}\n" for i, s in enumerate(reads)).encode()


def rc(s):
    return s[::-1].translate(str.maketrans("ACGTacgtN", "TGCAtgcaN"))


def edge_reads(k, seed):
    rng = np.random.default_rng(seed)
    g = "".join("ACGT"[c] for c in rng.integers(0, 4, 6000))
    lens = [k + 1, k + 2, k + 3, 63, 64, 65, 79, 80, 81, 127, 128, 129, 143, 150, 151, 250, 495, 496, 497, 511, 512, 513,
            514, 527, 528, 529, 1023, 1024, 1025, 2000, 5000]
    reads = []
    for L in [x for x in lens if x >= k + 1] * 3:
        p = int(rng.integers(0, len(g) - L + 1))
        s = g[p:p + L]
        reads.append(rc(s) if rng.random() < 0.5 else s)
    reads += [g[100:260]] * 5 + [rc(g[100:260])] * 4            # duplicates on both strands
    for unit in ("A", "T", "AC", "AAG", "ACGT", g[:20]):        # a minimizer that recurs
        reads += [(unit * 700)[:n] for n in (k + 2, 200, 700)]
    for n, at in ((150, 0), (150, 149), (150, 77), (600, 599), (1500, 3), (1500, 1499), (k + 2, 5)):
        s = list(g[300:300 + n])
        s[at] = "N"
        reads.append("".join(s))
    reads += [g[400:560].lower(), g[400:700].swapcase(), g[800:950], g[:k], g[:k - 1], "ACG"]
    return reads


@pytest.mark.parametrize("k", [19, 22, 23, 30, 31, 32, 33, 46, 47, 48, 62, 63])
def test_extraction_edges(k):
    data = fastq(edge_reads(k, k))
    for thr_on, thr in ((True, bg.thresholds([2])), (False, bg.thresholds())):
        ref = oracle.run(data, k=k, thresholding=thr_on, thresh=thr, min_update=True, keep_k2=True, keep_filtered=True)
        compare(gpu_run(data, k, thr_on, thr, True), ref)
    # the same reads in pieces of a host copy
    thr = bg.thresholds([2])
    ref = oracle.run(data, k=k, thresh=thr, min_update=True, keep_k2=True, keep_filtered=True)
    compare(gpu_run(data, k, True, thr, True, h2d_chunk=4096), ref)


def low_mmer(seed):
    """an M-mer of a very small order (kmer.cuh mz_order), so that it is the minimizer wherever it is"""
    x = np.random.default_rng(seed).integers(0, 1 << 30, 1 << 20).astype(np.uint64)
    r = np.zeros_like(x)
    y = x.copy()
    for _ in range(M):
        r = (r << np.uint64(2)) | (np.uint64(3) - (y & np.uint64(3)))
        y >>= np.uint64(2)
    m = np.uint64(0xFFFFFFFF)
    h = ((np.minimum(x, r) ^ np.uint64(0x2C9277B5)) * np.uint64(0x9E3779B1)) & m
    v = int(x[np.argmin(h)])
    return "".join("ACGT"[(v >> (2 * (M - 1 - i))) & 3] for i in range(M))


@pytest.mark.parametrize("k,n", [(31, 40), (31, 400), (31, 3000), (45, 150), (63, 400)])
def test_crowded_partition(k, n):
    """n places share one minimizer: their k-mers (k - 14 each) land in one partition, past its
    block's slots, past the larger block's, or neither"""
    rng = np.random.default_rng(n)
    mm = low_mmer(k)
    reads = []
    for _ in range(n):
        a, b = ("".join("ACGT"[c] for c in rng.integers(0, 4, 60)) for _ in range(2))
        reads += [a + mm + b, rc(a + mm + b)]
    data = fastq(reads)
    thr = bg.thresholds([2])
    ref = oracle.run(data, k=k, thresh=thr, min_update=True, keep_k2=True, keep_filtered=True)
    compare(gpu_run(data, k, True, thr, True), ref)


@pytest.mark.parametrize("lower", [1, 2, 5])
@pytest.mark.parametrize("k", [21, 31, 45])
def test_one_call_keeps_what_the_filter_keeps(k, lower):
    """bruno_build_and_compact leaves out of the table what the filter would drop: the graph, the
    counts and the flag histogram are the oracle's all the same, with k-mers of many biedges (a
    k-mer between every pair of bases) among them"""
    rng = np.random.default_rng(k * 10 + lower)
    core = "".join("ACGT"[c] for c in rng.integers(0, 4, k))
    wide = ["".join("ACGT"[c] for c in rng.integers(0, 4, 40)) + a + core + b +
            "".join("ACGT"[c] for c in rng.integers(0, 4, 40)) for a in "ACGT" for b in "ACGT"]
    data = fastq(edge_reads(k, 7) + wide * 3 + [core + w[50:] for w in wide])
    thr = bg.thresholds([lower])
    ref = oracle.run(data, k=k, thresh=thr, min_update=True)
    with bg.Graph(k=k, thresh=thr, min_update=True) as g:
        g.build_and_compact(data)
        s = g.sizes()
        for n in ("n_instances", "n_k2", "n_nodes", "n_branch", "n_chain_nodes", "iterations", "n_ranked", "n_chains"):
            assert s[n] == ref[n], (n, s[n], ref[n])
        assert s["filter_flag_hist"] == ref["filter_flag_hist"]
        assert_same(sort_nodes(*g.nodes()), ref["nodes"], "graph nodes")
        assert_same(sort_ranked(*g.ranked()), ref["ranked"], "listranked chain nodes")
        assert chain_set(*g.chains()) == chain_set(*ref["chains"])


@pytest.mark.parametrize("with_k1", [False, True])
@pytest.mark.parametrize("k", [20, 21, 31, 32, 45, 62, 63])
def test_edge_filter_from_the_entries(k, with_k1):
    """the (k+1)-mer filter of a one-call build: (k+1)-mers and (even k) k-mers that are their own
    reverse complements, homopolymers and k-mers between every pair of bases, with bounds around their
    counts; a read of k + 1 bases has a (k+1)-mer and no k-mer"""
    rng = np.random.default_rng(k)
    rand = lambda n: "".join("ACGT"[c] for c in rng.integers(0, 4, n))
    core, half = rand(k), rand((k + 1) // 2)
    wide = [rand(40) + a + core + b + rand(40) for a in "ACGT" for b in "ACGT"]
    pal = [rand(50) + half + rc(half) + rand(50) for _ in range(3)]
    reads = [r for r in edge_reads(k, 3) if with_k1 or len(r) != k + 1]
    reads += wide * 2 + pal * 2 + [rc(x) for x in pal] + [core + w[60:] for w in wide] + [half + rc(half) + "A", "A" * (k + 2)]
    if with_k1:
        reads += [(half + rc(half))[:k + 1], core + "A"] * 2
    data = fastq(reads)
    for lo, hi in ((1, 65536), (2, 65536), (5, 65536), (2, 9)):
        thr = np.array([0, 65536, lo, hi, 0, 65536], dtype=np.uint64)
        ref = oracle.run(data, k=k, thresh=thr, min_update=True, keep_k2=True, keep_filtered=True, edge_filter=True)
        compare_one_call(one_call_run(data, k, True, thr, True, edge_filter=True), ref)


@pytest.mark.parametrize("tiny", [0, 40])
def test_records_to_partitions_in_two_passes(tiny):
    """an input of more than 2^20 records (at most 17 k-mers each) in 2^12 partitions and more, alone and
    in a batch behind samples whose partitions hold next to nothing: a tile of records then spans more
    groups of partitions than it counts"""
    rng = np.random.default_rng(5)
    g = rng.integers(0, 4, 1_000_000)
    at = rng.integers(0, len(g) - 100, 270_000)
    codes = g[at[:, None] + np.arange(100)]
    err = rng.random(codes.shape) < 0.01
    codes = np.where(err, (codes + rng.integers(1, 4, codes.shape)) & 3, codes)
    text = np.frombuffer(b"ACGT", dtype=np.uint8)[codes]
    big = b"".join(b"@r\n" + row.tobytes() + b"\n+\n" + b"I" * 100 + b"\n" for row in text)
    thr = bg.thresholds([2])
    if not tiny:
        ref = oracle.run(big, k=31, thresh=thr, min_update=True, threads=16)
        with bg.Graph(k=31, thresh=thr, min_update=True) as gr:
            gr.build_and_compact(big)
            s = gr.sizes()
            assert s["n_instances"] >= 17 << 20 and s["table_partitions"] >= 1 << 12
            for n in ("n_instances", "n_k2", "n_nodes", "n_branch", "n_chain_nodes", "n_ranked", "n_chains"):
                assert s[n] == ref[n], (n, s[n], ref[n])
            assert_same(sort_nodes(*gr.nodes()), ref["nodes"], "graph nodes")
            assert chain_set(*gr.chains()) == chain_set(*ref["chains"])
        return
    lines = big.split(b"\n")
    small = [b"\n".join(lines[16 * i:16 * i + 16]) + b"\n" for i in range(tiny)]
    samples = small[:tiny // 2] + [big] + small[tiny // 2:]
    got, _ = batch(samples, k=31, thresholding=True, thresh=thr, min_update=True)
    for i in (0, tiny // 2 - 1, tiny // 2, tiny // 2 + 1, tiny):
        same_as_plain(got[i], plain(samples[i], k=31, thresholding=True, thresh=thr, min_update=True), f"sample {i}")


@pytest.mark.parametrize("k", [31, 63])
def test_partitions_of_four_bins_at_least(k):
    """partitions so small (256 and 128 slots) that the plan asks for more of them than a quarter of the
    bins: they get larger instead"""
    rng = np.random.default_rng(k)
    g = "".join("ACGT"[c] for c in rng.integers(0, 4, 200_000))
    reads = []
    for at in rng.integers(0, len(g) - 100, 30_000):
        s = list(g[at:at + 100])
        s[int(rng.integers(0, 100))] = "ACGT"[int(rng.integers(0, 4))]
        reads.append("".join(s))
    data = fastq(reads)
    thr = bg.thresholds([2])
    ref = oracle.run(data, k=k, thresh=thr, min_update=True, threads=16, keep_k2=True, keep_filtered=True)
    compare_one_call(one_call_run(data, k, True, thr, True, part_slots=256), ref)
    compare(gpu_run(data, k, True, thr, True, part_slots=256), ref)
