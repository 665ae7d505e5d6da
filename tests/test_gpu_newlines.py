"""Newline positions from the counting pass's bits (k_nl_place) and, where the budget has no room for the bits, from the
bytes again (k_nl_write): at every budget that lets a job count its reads the counts are those of a job without one."""
import numpy as np
import pytest

from metapart_gb300 import native, synth

pytestmark = pytest.mark.gpu


def _count(budget, data):
    with native.Context(0, budget) as ctx, native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(21, [0, len(data)])
        return cnt.hist.copy(), cnt.chunk_reads.copy()


@pytest.mark.parametrize("lengths", [(150,), (1, 22, 300), (300, 5)])
def test_bits_or_bytes(built_gpu, lengths):
    data = synth.fastq_bytes(synth.ReadSpec(120_000, lengths, 10, (20_000, 50_000), qual="I", seed=len(lengths)))
    want = _count(0, data)
    fits = []
    for percent in range(100, 220, 4):
        try:
            got = _count((len(data) * percent) // 100 + (12 << 20), data)
        except native.MetapartError as e:
            assert "memory" in str(e) or "budget" in str(e)
            fits.append(False)
            continue
        fits.append(True)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert fits[-1]


@pytest.mark.parametrize("n", [2, 208, 210, 1_000, 4_178])
def test_block_edges(built_gpu, n):
    """Inputs around the 65,536 bytes of a block: records' starts are found."""
    data = synth.fastq_bytes(synth.ReadSpec(n, (150,), 2, (5_000, 9_000), qual="I", seed=n))
    at = np.concatenate([[0], np.flatnonzero(np.frombuffer(bytes(data), np.uint8) == 10)[3::4] + 1])
    pick = np.unique(np.linspace(0, n, min(n, 50) + 1).astype(int))
    with native.Context(0) as ctx, native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(21, at[pick].astype(np.uint64))
        assert cnt.chunk_reads.tolist() == np.diff(pick).tolist()
