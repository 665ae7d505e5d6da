"""Component sizes counted by blocks in shared memory (k_sizes): the partition bounds, which are the prefix of the sizes,
follow from the labels.  Reads of a few components, of more small ones than a block's table has slots, of one giant one,
and more reads than one per thread."""
import numpy as np
import pytest

from metapart_gb300 import native, synth

pytestmark = pytest.mark.gpu

CASES = [(700, 2, 20_000), (60_000, 4, 40_000), (400_000, 40, 1_000_000), (400_000, 1, 100_000)]


@pytest.mark.parametrize("n,genomes,length", CASES, ids=lambda v: str(v))
def test_bounds_follow_from_labels(built_gpu, n, genomes, length):
    data = synth.fastq_bytes(synth.ReadSpec(n, (100,), genomes, (length, length), sub_rate=0.003, qual="I", seed=n + genomes))
    with native.Context(0) as ctx, native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(27, [0, len(data)])
        bounds = job.partition(27, 1, 1, [0, len(data)], cnt.chunk_first_read, cnt.hist)
        label = np.array(job.labels(), dtype=np.int64)
    read = np.arange(n)
    root = np.where(label == 0xFFFFFFFF, read, label)
    size = np.bincount(root, minlength=n)
    prefix = np.concatenate([[0], np.cumsum(np.where(label == read, size, 0))])
    want = [0] + [int(np.searchsorted(prefix, i * (n // 16))) for i in range(1, 16)] + [n]
    assert [int(x) for x in bounds] == want
