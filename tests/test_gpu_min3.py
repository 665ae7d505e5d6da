"""The 3-minimizer window loop (min3_read, eight bytes at a time) against the oracle: k on both sides of 17 (two code
paths), reads of k to k + 4 bases (windows of no or one position), every alignment of a read's first byte, Ns, and one
k-mer throughout (poly-A, whose code 0 the loop takes for no minimum)."""
import pytest

import pipeline_util as pu
from metapart_gb300 import synth

pytestmark = pytest.mark.gpu


def _odd_reads(k):
    recs = []
    for i in range(160):
        L = k + i % 23
        seq = bytes("ACGT"[(i * 7 + j * j + (j >> 2)) % 4].encode()[0] for j in range(L))
        if i % 5 == 0:
            seq = b"A" * L if i % 10 else seq[:L // 2] + b"N" + seq[L // 2 + 1:]
        recs.append(b"@" + b"x" * (1 + i % 9) + b"\n" + seq + b"\n+\n" + b"I" * L + b"\n")
    return b"".join(recs)


@pytest.mark.parametrize("k", [11, 16, 17, 28, 31])
def test_min3_matches_oracle(tmp_path, built_gpu, k):
    fq = tmp_path / "in.fastq"
    spec = synth.ReadSpec(6_000, (k + 1, 60, 101, 250), 6, (3_000, 30_000), sub_rate=0.01, n_rate=2e-3, seed=k)
    fq.write_bytes(_odd_reads(k) + synth.fastq_bytes(spec) + _odd_reads(k))
    p = pu.Params(k=k, chunks=4, scans=1, threads=2, min3=True)
    a = pu.outputs(pu.run("oracle", tmp_path, [fq], p), p, "in.fastq")
    for dump in (True, False):  # the sorted scans (their tuples dumped) and the grouped ones
        b = pu.outputs(pu.run("gpu", tmp_path, [fq], p, dump=dump), p, "in.fastq")
        keys = [x for x in a if not x.startswith("dump/")]
        if dump:
            keys += [f"dump/scan0_{w}.bin" for w in ("enum", "sorted", "filtered", "bad")]
        assert not [x for x in keys if x not in b]
        assert not pu.diff_keys(a, b, keys)
