"""A batch whose samples' reads have different lengths, so that each sample's reads are tiled by themselves in the first
split pass: every sample against the same sample alone."""
import pytest

from metapart_gb300 import native, synth
from test_gpu_batch import _batched, _check

pytestmark = pytest.mark.gpu

LENGTHS = [(40,), (250,), (31, 32, 33), (20,), (151, 76, 265), (100,)]


@pytest.mark.parametrize("k", [15, 31])
def test_samples_of_different_read_lengths(built_gpu, k):
    data = []
    for i, lengths in enumerate(LENGTHS):
        n = 700 + 260 * i
        mixed = lengths if max(lengths) > k else (*lengths, k + 9)  # (a sample without any k-mer is refused)
        data.append(synth.fastq_bytes(synth.ReadSpec(n, mixed, 3, (5_000, 20_000), sub_rate=0.005, n_rate=1e-3, qual="#J",
                                                     seed=40 + i)))
    shapes = [(2, 2), (1, 1), (4, 2), (2, 1), (4, 4), (1, 1)]
    with native.Context(0) as ctx:
        res, outs, fs, labs, _ = _batched(ctx, data, shapes, k)
        _check(ctx, data, shapes, k, res, outs, fs, labs)
