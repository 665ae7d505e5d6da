"""The path that runs by default (grouped scans) against the CPU oracle, byte for byte, at the parity cases: the partition
files without any dump, the per-read dumps (BAD flags, parents after every scan), and with the self-checks, which run every
scan both ways and compare.
"""
import pytest

import pipeline_util as pu
from metapart_gb300 import native, synth
from test_gpu_parity import CASES, _keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n,p", CASES, ids=[f"{c[0]}-{c[1]}-k{c[2].k}-s{c[2].scans}-t{c[2].threads}" for c in CASES])
def test_grouped_matches_oracle(tmp_path, built_gpu, name, n, p):
    fq = tmp_path / "in.fastq"
    synth.write_fastq(synth.workload(name, n, seed=12), fq)
    want = pu.outputs(pu.run("oracle", tmp_path, [fq], p), p, "in.fastq")
    every = _keys(want, p)
    reads = [x for x in every if not x.startswith("dump/scan") or x.endswith("_bad.bin")]
    files = [x for x in every if not x.startswith("dump/")]
    for keys, dump, env in ((files, False, None), (reads, True, {"MP_DUMP_TUPLES": "0"}), (every, True, {"MP_CHECK": "1"})):
        got = pu.outputs(pu.run("gpu", tmp_path, [fq], p, dump=dump, env_extra=env), p, "in.fastq")
        assert not [x for x in keys if x not in got]
        assert not pu.diff_keys(want, got, keys), env


@pytest.fixture(scope="module")
def ctx(built_gpu):
    c = native.Context(0)
    yield c
    c.close()


def _launches(ctx, data, scans, min3, checks, dump_dir=None):
    fno, ofs = native.fastq_index(4, [data])
    starts = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Job(ctx) as job:
        job.set_checks(checks)
        job.set_dump_dir(dump_dir)
        job.load(data)
        cnt = job.count(31, starts, min3)
        before = native.launch_count()
        job.partition(31, scans, 2, starts, cnt.chunk_first_read, cnt.hist, min3)
        return native.launch_count() - before, job.sort_split()["unit_passes"]


@pytest.mark.parametrize("scans,min3", [(1, False), (2, False), (1, True)])
def test_checks_run_the_grouped_scans(ctx, tmp_path, scans, min3, monkeypatch):
    """A checked job makes the launches of the grouped scans beside those of the sorted ones; per-read dumps leave the scans
    grouped, tuple dumps do not."""
    data = synth.fastq_bytes(synth.workload("plain_large", 20_000, seed=4))
    grouped, passes = _launches(ctx, data, scans, min3, False)
    assert passes == 0
    sorted_, passes = _launches(ctx, data, scans, min3, False, tmp_path)
    assert passes > 0
    both, _ = _launches(ctx, data, scans, min3, True)
    assert both > sorted_ + 10 * scans and both > grouped + 10 * scans
    monkeypatch.setenv("MP_DUMP_TUPLES", "0")
    assert _launches(ctx, data, scans, min3, False, tmp_path)[1] == 0
