"""bruno_build_samples with one sample: the plain build's results through the batch's calls."""
import numpy as np
import pytest

import bruno_gb300 as bg
from conftest import fixture_bytes
from test_gpu_batch import batch, mixed_samples, plain, same_as_plain
from test_gpu_superkmer_limits import crowded_reads, fastq

pytestmark = pytest.mark.gpu

CFG = dict(thresholding=True, thresh=bg.thresholds([2]), min_update=True)


@pytest.mark.parametrize("k", [17, 21, 31])
@pytest.mark.parametrize("data", ["natural.withN.fastq", "debruijn.shifted_cycle_chr14.fastq", "crowded", "empty"])
def test_batch_of_one(data, k):
    data = b"" if data == "empty" else fastq(crowded_reads("adapter", 2)) if data == "crowded" else fixture_bytes(data)
    got, total = batch([data], k=k, **CFG)
    p = plain(data, k=k, **CFG)
    same_as_plain(got[0], p, "sample 0")
    assert total["n_chains"] == p["sizes"]["n_chains"]


def test_between_batches_and_plain_builds():
    """one context: a batch, a batch of one, a plain build (no batch any more), a batch again"""
    samples = mixed_samples()
    with bg.Graph(k=31, **CFG) as g:
        for group in (samples, samples[:1], samples[3:4], samples):
            g.build_samples(group)
            assert g.sample_count() == len(group)
            for i, data in enumerate(group):
                want = plain(data, k=31, **CFG)["sizes"]
                got = g.sample_sizes(i)
                assert all(got[n] == want[n] for n in ("n_reads", "n_k2", "n_nodes", "n_chains", "n_chain_chars")), i
        g.build_and_compact(samples[0])
        with pytest.raises(bg.BrunoError):
            g.sample_sizes(0)
        g.build_samples(samples[:1])
        with pytest.raises(bg.BrunoError):
            g.clean_deadend_and_bubbles_naive()


def test_one_sample_in_device_memory():
    import torch
    data = mixed_samples()[0]
    d = torch.from_numpy(np.frombuffer(bytes(data), dtype=np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    with bg.Graph(k=31, **CFG) as g:
        g.build_samples([d.data_ptr()], is_device=True, nbytes=[d.numel()])
        want = plain(data, k=31, **CFG)["sizes"]
        assert g.sample_sizes(0)["n_chains"] == want["n_chains"] == g.sizes()["n_chains"]
