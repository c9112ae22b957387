"""Which counting path runs, and the one by k-mer records at the lengths where super-k-mers run by
default: an explicit table size keeps it (a batch takes no notice of the size itself)."""
import numpy as np
import pytest

import bruno_gb300 as bg
from bruno_gb300 import synth
from conftest import fixture_bytes
from helpers import assert_same, chain_set, sort_nodes
from oracle import oracle
from test_gpu_batch import batch, mixed_samples, plain, same_as_plain
from test_gpu_parity import FASTQS, OPTIONS, compare, compare_one_call, gpu_run, one_call_run
from test_gpu_superkmer_limits import fastq, rand_reads

pytestmark = pytest.mark.gpu


def path_of(data, k, **cfg):
    with bg.Graph(k=k, thresh=bg.thresholds([2]), min_update=True, **cfg) as g:
        g.build_and_compact(data)
        return g.counting_path()


@pytest.mark.parametrize("k,cfg,want", [
    (17, {}, "kmer_records"), (18, {}, "kmer_records"), (19, {}, "super_kmers"), (31, {}, "super_kmers"),
    (32, {}, "super_kmers"), (63, {}, "super_kmers"), (31, {"table_slots": 1 << 20}, "kmer_records"),
    (63, {"table_slots": 1 << 20}, "kmer_records"), (31, {"direct_count": 2}, "l2_partitions"),
    (31, {"direct_count": 1}, "whole_table"), (63, {"direct_count": 1}, "whole_table"),
    (31, {"edge_filter": True}, "super_kmers"), (31, {"edge_filter": True, "keep_k2": True}, "kmer_records")])
def test_path(k, cfg, want):
    rng = np.random.default_rng(k)
    reads = rand_reads(rng, rng.integers(0, 4, 20_000), 4_000, 100, 0.005)
    path, records = path_of(fastq(reads), k, **cfg)
    assert path == want
    instances = len(reads) * (100 - k + 1)
    if path in ("kmer_records", "l2_partitions"):
        assert records == instances
    elif path == "super_kmers":
        assert len(reads) <= records
    else:
        assert records == 0


@pytest.mark.parametrize("k,least", [(22, False), (23, False), (24, True), (26, True), (27, True)])
def test_path_where_every_kmer_is_kept(k, least):
    """steps, raw counts and unthresholded builds of more than 2 MB by k-mer records below k = 24 (27 with a
    target load above 0.6), thresholded builds in one call and small ones by super-k-mers; the same graph"""
    rng = np.random.default_rng(k)
    data = fastq(rand_reads(rng, rng.integers(0, 4, 60_000), 12_000, 100, 0.005))
    assert len(data) > 2 << 20
    want = "super_kmers" if least else "kmer_records"
    assert path_of(data, k)[0] == "super_kmers"
    assert path_of(data, k, keep_k2=True)[0] == want
    assert path_of(data, k, thresholding=False)[0] == want
    assert path_of(data, k, thresholding=False, max_load=0.7)[0] == ("super_kmers" if k >= 27 else "kmer_records")
    assert path_of(data[:207 * 9_000], k, thresholding=False)[0] == "super_kmers"   # (207 bytes a record)
    with bg.Graph(k=k, thresh=bg.thresholds([1]), min_update=True) as g:   # (bounds that drop nothing)
        g.build_and_compact(data)
        assert g.counting_path()[0] == want
    thr = bg.thresholds([2])
    ref = oracle.run(data, k=k, thresh=thr, min_update=True, threads=16, keep_k2=True, keep_filtered=True)
    compare(gpu_run(data, k, True, thr, True), ref)


@pytest.mark.parametrize("chunk", [0, 1 << 20])
@pytest.mark.parametrize("length,want", [(36, "kmer_records"), (50, "super_kmers"), (300, "super_kmers")])
def test_path_by_the_reads_lengths(length, want, chunk):
    """an unthresholded build at k = 31: reads of six k-mers go by k-mer records, at once and in pieces of a
    host copy, whose first piece says; with thresholds they do not"""
    rng = np.random.default_rng(length)
    data = fastq(rand_reads(rng, rng.integers(0, 4, 60_000), 4_000_000 // length, length, 0.005))
    assert path_of(data, 31, thresholding=False, h2d_chunk=chunk)[0] == want
    assert path_of(data, 31, h2d_chunk=chunk)[0] == "super_kmers"
    ref = oracle.run(data, k=31, thresholding=False, thresh=bg.thresholds(), min_update=True, threads=16, keep_k2=True,
                     keep_filtered=True)
    compare(gpu_run(data, 31, False, bg.thresholds(), True, h2d_chunk=chunk), ref)


def test_path_is_forgotten():
    with bg.Graph(k=31, thresh=bg.thresholds([2]), min_update=True) as g:
        assert g.counting_path() == ("none", 0)
        g.build_and_compact(fixture_bytes("natural.fastq"))
        assert g.counting_path()[0] == "super_kmers"
        g.reset()
        assert g.counting_path() == ("none", 0)


@pytest.mark.parametrize("opt", sorted(OPTIONS))
@pytest.mark.parametrize("fname", FASTQS)
def test_kmer_records_fixture_parity(fname, opt):
    thr_on, lo, mu = OPTIONS[opt]
    thr = bg.thresholds(lo)
    data = fixture_bytes(fname)
    ref = oracle.run(data, k=31, thresholding=thr_on, thresh=thr, min_update=mu, keep_k2=True, keep_filtered=True)
    compare(gpu_run(data, 31, thr_on, thr, mu, table_slots=1 << 18), ref)


@pytest.mark.parametrize("chunk", [0, 4 << 20])
@pytest.mark.parametrize("k", [21, 31, 45, 63])
def test_kmer_records_workload_parity(k, chunk):
    """the steps and one call, at once and in pieces of a host copy (extracted as they land at k <= 31)"""
    w = synth.Workload("records", 400_000, 100, 60_000, 0.01, k, (2,), 0.03, (500, 4000), (2, 6), (0.01, 0.02), 4)
    data = bytes(synth.make_fastq(w))
    thr = bg.thresholds(w.lower)
    ref = oracle.run(data, k=k, thresh=thr, min_update=True, threads=16, keep_k2=True, keep_filtered=True)
    compare(gpu_run(data, k, True, thr, True, table_slots=1 << 23, h2d_chunk=chunk), ref)
    compare_one_call(one_call_run(data, k, True, thr, True, table_slots=1 << 23, h2d_chunk=chunk), ref)
    assert path_of(data, k, table_slots=1 << 23, h2d_chunk=chunk)[0] == "kmer_records"


@pytest.mark.parametrize("k", [31, 45])
def test_kmer_records_edge_filter(k):
    """(a k-mer that crowds a hash bucket is refused under this filter at k <= 31)"""
    rng = np.random.default_rng(k)
    data = fastq(rand_reads(rng, rng.integers(0, 4, 120_000), 24_000, 100, 0.003))
    thr = bg.thresholds([3])
    ref = oracle.run(data, k=k, thresh=thr, min_update=True, threads=16, edge_filter=True, keep_k2=True, keep_filtered=True)
    compare_one_call(one_call_run(data, k, True, thr, True, edge_filter=True, table_slots=1 << 22), ref)


@pytest.mark.parametrize("chunk", [0, 256 << 10])
def test_kmer_records_in_a_batch(chunk):
    samples = mixed_samples()
    cfg = dict(k=31, thresholding=True, thresh=bg.thresholds([2]), min_update=True)
    got, _ = batch(samples, table_slots=1, h2d_chunk=chunk, **cfg)
    for i, data in enumerate(samples):
        same_as_plain(got[i], plain(data, **cfg), f"sample {i}")
    with bg.Graph(table_slots=1, h2d_chunk=chunk, **cfg) as g:
        g.build_samples(samples)
        assert g.counting_path()[0] == "kmer_records"


@pytest.mark.parametrize("k", [31, 45])
def test_exact_counts_past_what_an_entry_holds(k):
    """300 bases a read, all alike, counted more than 2^26 times in all: by super-k-mers whether the counts
    are copied out or not, to the last occurrence"""
    n = (1 << 26) // (300 - k - 1) + 2000
    data = fastq(np.zeros((n, 300), dtype=np.int8))
    assert path_of(data, k)[0] == "super_kmers"
    with bg.Graph(k=k, thresh=bg.thresholds([2]), min_update=True, keep_k2=True, keep_filtered=True) as g:
        g.build_and_compact(data)
        assert g.counting_path()[0] == "super_kmers"
        for keys, edges, counts in (g.k2(), g.filtered()):
            assert int(counts.max()) == n * (300 - k - 1) and counts.dtype == np.uint32
        assert int(g.k2()[2].sum()) == n * (300 - k + 1)


@pytest.mark.parametrize("steps", [False, True])
def test_second_attempt_over_records_in_order(steps):
    """a table too small for what is kept (a target load above one) after the records went to their
    partitions in two passes: the second attempt's plan orders them again"""
    rng = np.random.default_rng(12)
    data = fastq(rand_reads(rng, rng.integers(0, 4, 1_000_000), 270_000, 100, 0.01))
    thr = bg.thresholds([2])
    ref = oracle.run(data, k=31, thresh=thr, min_update=True, threads=16)
    with bg.Graph(k=31, thresh=thr, min_update=True, part_slots=256, max_load=3.0) as g:
        if steps:
            g.load_fastq(data)
            g.compute_biedge_freqencies()
            g.local_insert_by_freqencies()
            g.extract_chains()
            g.list_rank_min_update()
            g.to_compressed_chains()
        else:
            g.build_and_compact(data)
        path, records = g.counting_path()
        assert path == "super_kmers" and records > 1 << 20 and g.sizes()["table_partitions"] >= 1 << 12
        assert_same(sort_nodes(*g.nodes()), ref["nodes"], "graph nodes")
        assert chain_set(*g.chains()) == chain_set(*ref["chains"])


def test_a_bin_past_its_tally():
    """more than 2^26 records of one minimizer (8.6M reads of 150 A): by other records, with the same graph; a
    batch with such a sample is declined, as its hash bucket always was, and the context builds on"""
    import torch
    reads, length, k = 8_600_000, 150, 31
    rec = fastq(np.zeros((100, length), dtype=np.int8))
    d = torch.from_numpy(np.frombuffer(rec, dtype=np.uint8).copy()).cuda().repeat(reads // 100)
    torch.cuda.synchronize()
    rng = np.random.default_rng(9)
    small = fastq(rand_reads(rng, rng.integers(0, 4, 20_000), 4_000, 100, 0.005))
    e = torch.from_numpy(np.frombuffer(small, dtype=np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    want = plain(small, k=k, thresh=bg.thresholds([2]), min_update=True)["sizes"]
    with bg.Graph(k=k, thresh=bg.thresholds([2]), min_update=True) as g:
        g.build_and_compact(d.data_ptr(), d.numel(), is_device=True)
        s = g.sizes()
        assert g.counting_path()[0] in ("l2_partitions", "whole_table")
        assert s["n_instances"] == reads * (length - k + 1) and s["n_k2"] == 3 and s["n_nodes"] == 1
        with pytest.raises(bg.BrunoError) as err:
            g.build_samples([e.data_ptr(), d.data_ptr()], is_device=True, nbytes=[e.numel(), d.numel()])
        assert err.value.status == 4
        g.build_samples([e.data_ptr(), e.data_ptr()], is_device=True, nbytes=[e.numel(), e.numel()])
        for i in range(2):
            assert all(g.sample_sizes(i)[n] == want[n] for n in ("n_k2", "n_nodes", "n_chains", "n_chain_chars"))


@pytest.mark.parametrize("chunk", [0, 1 << 20])
@pytest.mark.parametrize("k,want", [(21, "kmer_records"), (31, "super_kmers")])
def test_path_of_an_unthresholded_batch(k, want, chunk):
    """samples of more than 2 MB on average, every k-mer kept, in one copy and in groups"""
    rng = np.random.default_rng(k)
    samples = [fastq(rand_reads(rng, rng.integers(0, 4, 40_000), n, 100, 0.005)) for n in (16_000, 9_000, 12_000)]
    cfg = dict(k=k, thresholding=False, min_update=True)
    got, _ = batch(samples, h2d_chunk=chunk, **cfg)
    for i, data in enumerate(samples):
        same_as_plain(got[i], plain(data, **cfg), f"sample {i}")
    with bg.Graph(h2d_chunk=chunk, **cfg) as g:
        g.build_samples(samples)
        assert g.counting_path()[0] == want
