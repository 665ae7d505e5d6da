"""Device memory of scans that are split together: the split tuples of all scans go back when a partition fails.
"""
import pytest

from metapart_gb300 import native, synth

pytestmark = pytest.mark.gpu


def _starts(data, chunks=4):
    fno, ofs = native.fastq_index(chunks, [data])
    return native.chunk_starts_of(fno, ofs, [len(data)])


def test_failed_partition_keeps_no_split_tuples(built_gpu):
    data = synth.fastq_bytes(synth.workload("hotspot", 40_000, seed=31))
    st = _starts(data)
    with native.Context(0) as ctx, native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(27, st)
        tuples = int(cnt.hist[-1])
        used = []
        for _ in range(3):
            job.set_wait_limits(union_retries=1)
            with pytest.raises(native.MetapartError, match="union-find"):
                job.partition(27, 2, 4, st, cnt.chunk_first_read, cnt.hist)
            used.append(ctx.hbm_in_use())
        assert used[2] - used[0] < 1 << 20 < 12 * tuples
        job.set_wait_limits()
        job.partition(27, 2, 4, st, cnt.chunk_first_read, cnt.hist)
