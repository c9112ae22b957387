"""bench.py's roofline rows follow the counting path that the library says it took."""
import importlib.util
import os

import pytest

from conftest import ROOT

SIZES = {"n_instances": 1000, "n_reads": 10, "n_nodes": 300, "table_slots": 700, "filter_slots_read": 400,
         "table_partitions": 1 << 18}
MS = {"count_estimate": 2.0, "count_insert": 7.0, "count_split": 3.0, "filter_insert": 1.0}


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("k,path,records,want", [
    (31, "super_kmers", 2 << 20, {"k_sk_extract": 5160 + 32 * (1 << 20), "k_sk_split": 64 * (1 << 20),
                                  "k_sk_count<KW1>": 32 * (1 << 20) + 32 * 700}),
    (63, "super_kmers", 100, {"k_sk_extract": 5160 + 3200, "k_sk_scatter": 6400, "k_sk_count<KW2>": 3200 + 64 * 700}),
    (31, "kmer_records", 1000, {"k_extract_s": 5160 + 8000, "k_split": 16000, "k_count_local": 8000 + 32 * 700 + 1600,
                                "k_filter": 32 * 700}),
    (63, "kmer_records", 1000, {"k_extract_s": 5160 + 16000, "k_split_scatter": 32000,
                                "k_count_local2": 16000 + 64 * 700 + 1600, "k_filter": 64 * 700}),
    (31, "l2_partitions", 1000, {"k_insert": 64000, "k_filter": 32 * 700}),
    (63, "whole_table", 0, {"k_count": 128000, "k_filter": 64 * 700})])
def test_rows(bench, k, path, records, want):
    got = bench.counting_kernels(k, path, records, 5000, SIZES, MS.__getitem__)
    assert {n: b for n, (b, _) in got.items()} == want
    assert sum(ms for _, ms in got.values()) == (9.0 if path == "super_kmers" else 10.0 if path == "kmer_records" else 8.0)
