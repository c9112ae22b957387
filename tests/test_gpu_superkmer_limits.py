"""Super-k-mer builds where an input outgrows what its plan foresaw, against the oracle and against the
plain build: more records than their room, cycles within one block of chain nodes, pointers that disagree."""
import numpy as np
import pytest

import bruno_gb300 as bg
from helpers import assert_same, chain_set, compress_ranked, sort_nodes, sort_ranked
from oracle import oracle
from test_gpu_batch import batch, plain, same_as_plain

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


def check(data, k, thr, thresholding=True, **cfg):
    """a one-call build against the oracle; returns its sizes"""
    ref = oracle.run(data, k=k, thresholding=thresholding, thresh=thr, min_update=True, threads=16,
                     edge_filter=cfg.get("edge_filter", False))
    with bg.Graph(k=k, thresholding=thresholding, thresh=thr, min_update=True, **cfg) as g:
        g.build_and_compact(data)
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
