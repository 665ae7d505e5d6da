"""The mate union's tail (one cluster of blocks, waiting pairs asleep) and the output plan's stable partition against
the oracle at the sizes where they change: one block and more of a cluster (1,024 pairs), launched rounds first
(above 24,576 pairs), the last unit of an output block full, short or of one (1,024 units of one or two reads).

The reads give the mate union what its rounds part on: components around the 1,000-read limit, many small ones, singles
beside both, and BAD reads; the labels, sizes and all partition files are compared byte for byte.
"""
import numpy as np
import pytest

import pipeline_util as pu
from metapart_gb300 import native, synth
from test_gpu_batch import _batched, _check

pytestmark = pytest.mark.gpu

PAIRS = [(1, False), (3, True), (511, False), (1023, False), (1024, True), (1025, False), (2049, True), (24_576, False),
         (24_577, False), (40_000, True)]


def _spec(n, il):
    g = max(2, n // 1500)  # log-normal abundances: from a few reads of a genome to several thousand
    return synth.ReadSpec(n, (100,), g, (20_000, 120_000), abundance=synth.AB_LOGNORMAL, ab_param=1.2, sub_rate=0.01,
                          n_rate=1e-4, interleaved=il, insert_len=280 if il else 0, seed=n)


@pytest.mark.parametrize("pairs,il", PAIRS)
def test_mate_union_and_output_match_oracle(tmp_path, built_gpu, pairs, il):
    fq = tmp_path / "in.fastq"
    synth.write_fastq(_spec(2 * pairs, il), fq)
    p = pu.Params(k=27, chunks=4 if pairs > 8 else 1, scans=1, threads=2 if pairs > 8 else 1, interleaved=il)
    a = pu.outputs(pu.run("oracle", tmp_path, [fq], p), p, "in.fastq")
    b = pu.outputs(pu.run("gpu", tmp_path, [fq], p), p, "in.fastq")
    keys = [k for k in a if not k.startswith("dump/")] + [f"dump/stats{s}_{w}.bin" for s in (1, 2) for w in ("parent", "sizes")]
    assert not [k for k in keys if k not in b]
    assert not pu.diff_keys(a, b, keys)


def test_mate_union_and_output_in_a_batch(built_gpu):
    data = [synth.fastq_bytes(_spec(2 * n, False)) for n in (1, 300, 1024, 24_577, 5, 2049)]
    shapes = [(1, 1), (2, 2), (4, 1), (8, 4), (1, 1), (4, 2)]
    with native.Context(0) as ctx:
        res, outs, fs, labs, _ = _batched(ctx, data, shapes, 27)
        _check(ctx, data, shapes, 27, res, outs, fs, labs)


def test_output_copies_records_of_all_lengths(built_gpu):
    """Records of 60 to 2,700 bytes (one turn of a warp and several) at every alignment: each file holds its records whole
    and in input order, and together they are the input."""
    rng = np.random.default_rng(3)
    recs = []
    for i in range(6_000):
        L = int(rng.integers(20, 270))
        seq = bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), L))
        name = b"@%d " % i + b"h" * int(rng.integers(0, 40) if i % 3 else rng.integers(0, 2_100))
        recs.append(name + b"\n" + seq + b"\n+\n" + b"I" * L + b"\n")
    data = b"".join(recs)
    with native.Context(0) as ctx, native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(21, [0, len(data)])
        job.partition(21, 1, 1, [0, len(data)], cnt.chunk_first_read, cnt.hist)
        out, sizes = job.output()
    at, seen = 0, []
    for size in sizes:
        part, last = bytes(out[at:at + int(size)]), -1
        at += int(size)
        while part:
            i = int(part[1:part.index(b" ")])
            assert i > last and part.startswith(recs[i])
            part, last = part[len(recs[i]):], i
            seen.append(i)
    assert at == len(data) and sorted(seen) == list(range(len(recs)))
