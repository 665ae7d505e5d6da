"""The work that users of this framework have it do, as cases that can be timed.

A case is one whole call chain through the public entry points: a partition job (chunk index, load, count,
partition, partition files), a batch of samples, a round of the request loop, or a tuple sort on device
pointers.  The read sets are the seeded synthetic ones of metapart_gb300.synth, whose shapes the tests and
the benchmark use.
"""
import math

import numpy as np
import torch

from metapart_gb300 import native, serve, synth


def _job(name, work, reads, length, genomes, k, scans, threads, chunks, store, io, **more):
    return dict(name=name, kind="job", work=work, reads=reads, length=length, genomes=genomes, k=k, scans=scans,
                threads=threads, chunks=chunks, store=store, io=io, **more)


def listed():
    return [
        # the smallest calls: a control sample or a test run, where launches and host round trips are the time
        _job("job 600 reads", "small", 600, 100, 20, 27, 1, 2, 4, "kmer_cache", "host"),
        # the smallest request of the serving mix
        _job("job 10k", "meta", 10_000, 150, 12, 31, 1, 16, 64, "packed", "host"),
        # the benchmark's small workload
        _job("job 100k k27", "small", 100_000, 100, 20, 27, 1, 16, 64, "kmer_cache", "host"),
        # trimmed reads of several lengths, some too short for a k-mer, three scans, no store of the reads
        # (the drop-in programs count and partition in two processes)
        _job("job ragged 151k 3 scans", "ragged", 151_162, 151, 23, 29, 3, 6, 30, "fastq", "host"),
        # interleaved pairs
        _job("job pairs 240k", "pairs", 240_000, 100, 40, 27, 2, 8, 32, "kmer_cache", "host"),
        # a viral or plasmid panel: few short genomes at a few thousand-fold coverage, long runs of one k-mer
        _job("job panel 300k", "panel", 300_000, 150, 30, 31, 1, 16, 64, "kmer_cache", "host"),
        # an ordinary sample of the serving and batch mixes
        _job("job 1M 2 scans", "meta", 1_000_000, 150, 30, 31, 2, 16, 64, "kmer_cache", "host"),
        # the 3-minimizer variant (a giant component), reads already on the GPU
        _job("job 3-minimizer 3M", "min3", 3_000_000, 250, 100, 31, 1, 16, 64, "fastq", "device"),
        # the benchmark's default workload, reads already on the GPU
        _job("job 20M 2 scans", "meta", 20_000_000, 150, 200, 31, 2, 16, 64, "kmer_cache", "device"),
        # many samples of uneven sizes and read lengths in one call
        dict(name="batch of 24", kind="batch", samples=24, lo=5_000, hi=400_000, k=31, threads=16, chunks=64),
        # the request loop with more requests than slots
        dict(name="request loop 12", kind="serve", requests=12, slots=8, lo=10_000, hi=600_000, k=31),
        # the tuple sort for callers with their own device arrays
        dict(name="sort 24M tuples", kind="sort", n=24_000_011, k=31, distinct=0.2, fixed=False),
    ]


def _even(x):
    return max(2, int(x) // 2 * 2)


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["job"] * 6 + ["batch", "serve", "sort", "sort"])
    if kind == "batch":
        lo = int(_log(rng, 1_000, 50_000))
        return dict(kind="batch", samples=rng.randint(3, 32), lo=lo, hi=lo * rng.randint(2, 8), k=rng.choice([21, 27, 31]),
                    threads=rng.choice([1, 4, 16]), chunks=32)
    if kind == "serve":
        lo = int(_log(rng, 5_000, 50_000))
        return dict(kind="serve", requests=rng.randint(4, 16), slots=rng.choice([1, 4, 8]), lo=lo,
                    hi=lo * rng.randint(2, 12), k=rng.choice([27, 31]))
    if kind == "sort":
        fixed = rng.random() < 0.5
        return dict(kind="sort", n=int(_log(rng, 1_000, 1_000_000 if fixed else 60_000_000)),
                    k=rng.choice([15, 21, 27, 28, 29, 31]), distinct=round(rng.uniform(0.01, 1.0), 3), fixed=fixed)
    work = rng.choice(["small", "meta", "meta", "ragged", "pairs", "panel", "min3"])
    io = rng.choice(["host", "device"])
    if work == "ragged":
        io = "host"
    reads = _even(_log(rng, 600, 2_500_000 if io == "host" else 10_000_000))
    if work == "panel":
        reads = min(reads, 1_000_000)
    threads = rng.choice([1, 2, 4, 16])
    c = _job("", work, reads, rng.choice([76, 100, 125, 150, 151, 250]), rng.randint(5, 120), rng.choice([19, 21, 25, 27, 28, 31]),
             1 if work == "min3" else rng.choice([1, 1, 2, 3]), threads, threads * (1 if reads < 5_000 else rng.randint(1, 4)),
             rng.choice(["kmer_cache", "kmer_cache", "packed", "fastq"]), io)
    if c["length"] == 250:
        c["reads"] = min(c["reads"], 6_000_000)
    del c["name"]
    return c


def _spec(c, seed):
    n, length, g = c["reads"], (c["length"],), c["genomes"]
    if c["work"] == "small":
        return synth.ReadSpec(n, length, g, (50_000, 50_000), sub_rate=0.005, qual="I", seed=seed)
    if c["work"] == "meta":
        return synth.ReadSpec(n, length, g, (1e6, 5e6), (0.3, 0.7), synth.AB_LOGNORMAL, 1.5, sub_rate=0.01, n_rate=1e-4,
                              qual="#J", seed=seed)
    if c["work"] == "ragged":
        top = c["length"]
        return synth.ReadSpec(n, (c["k"] - 4, max(c["k"], top // 2), max(c["k"], 2 * top // 3), top), g, (2e4, 4e5), (0.35, 0.65),
                              synth.AB_LOGNORMAL, 1.5, sub_rate=0.01, n_rate=1e-3, qual="#J", seed=seed)
    if c["work"] == "pairs":
        return synth.ReadSpec(n, length, g, (40_000, 400_000), sub_rate=0.005, qual="#J", interleaved=True,
                              insert_len=2 * c["length"] + 80, seed=seed)
    if c["work"] == "panel":
        return synth.ReadSpec(n, length, g, (3_000, 30_000), (0.35, 0.65), synth.AB_LOGNORMAL, 1.0, sub_rate=0.003,
                              qual="I", seed=seed)
    return synth.ReadSpec(n, length, g, (2e6, 2e6), abundance=synth.AB_ZIPF, ab_param=1.1, repeat_frac=0.3, repeat_len=5000,
                          repeat_pool=200, sub_rate=0.01, qual="I", seed=seed)


def _pinned(nbytes):
    t = torch.empty(int(nbytes), dtype=torch.uint8, pin_memory=True)
    return t, t.data_ptr()


def _mix(specs, seed):
    """The read sets of a mix: its sizes are the mix's own, its genomes and reads the seed's."""
    for i, x in enumerate(specs):
        x.seed = (1 + seed) * 1000 + i
    return [synth.fastq_to(x, _pinned) for x in specs]


class _State:
    """What a program keeps: the context, its job, batch or server, and its buffers."""

    def __init__(self, case):
        self.case = case
        self.ctx = native.Context(0)
        self.held = []

    def keep(self, x):
        self.held.append(x)
        return x

    def __del__(self):
        for x in reversed(self.held):
            x.close()
        self.ctx.close()


class _Bytes:
    """Device bytes at an address, for torch."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 2}


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind == "job":
        s.il = case["work"] == "pairs"
        s.host = synth.fastq_to(_spec(case, 1 + seed), _pinned)
        s.n = s.host.numel()
        s.job = s.keep(native.Job(s.ctx))
        s.job.set_read_store(case["store"])
        if case["io"] == "device":  # a caller whose reads are on the GPU has their chunk index from the load
            fno, ofs = native.fastq_index_ptr(case["chunks"], s.host.data_ptr(), s.n, s.il)
            s.starts = native.chunk_starts_of(fno, ofs, [s.n])
            s.dev = torch.zeros(s.n + 64, dtype=torch.uint8, device="cuda")
            s.dev[:s.n].copy_(s.host)
            s.host = None
        else:
            s.out = _pinned(case["reads"] * (2 * case["length"] + 6 + 10) + 64)[0].zero_()
    elif kind == "batch":
        s.batch = s.keep(native.Batch(s.ctx))
        s.hosts = _mix(synth.batch_mix(case["samples"], 5, case["lo"], case["hi"]), seed)
        s.outs = [_pinned(h.numel() + 64)[0] for h in s.hosts]
    elif kind == "serve":
        s.server = s.keep(serve.Server(s.ctx, case["slots"], 160 << 30))
        s.hosts = _mix(synth.serving_mix(case["requests"], 11, case["lo"], case["hi"]), seed)
        s.outs = [_pinned(h.numel() + 64)[0] for h in s.hosts]
        s.params = serve.RequestParams(k=case["k"])
    else:
        g = torch.Generator(device="cuda").manual_seed(1 + seed)
        n, k = case["n"], case["k"]
        pool = torch.randint(0, 1 << (2 * k), (max(1, int(n * case["distinct"])),), generator=g, device="cuda")
        kmer = pool[torch.randint(0, pool.numel(), (n,), generator=g, device="cuda")]
        adj = torch.randint(0, 64, (n,), generator=g, device="cuda")
        s.lo = (kmer << 8) | adj
        s.hi = (kmer >> 56).to(torch.uint8) if 2 * k + 8 > 64 else None
        s.id = torch.randint(0, 1 << 24, (n,), generator=g, device="cuda").to(torch.int32)
        s.lo2, s.id2 = torch.empty_like(s.lo), torch.empty_like(s.id)
        s.hi2 = torch.empty_like(s.hi) if s.hi is not None else None
    return s


def _run_job(s):
    c, job = s.case, s.job
    k, m3 = c["k"], c["work"] == "min3"
    job.reset()
    if c["io"] == "device":
        job.load_device_inplace(s.dev.data_ptr(), s.n, interleaved=s.il)
        cnt = job.count(k, s.starts, m3)
        bounds = job.partition(k, c["scans"], c["threads"], s.starts, cnt.chunk_first_read, cnt.hist, m3)
        sizes = np.zeros(16 * c["threads"], dtype=np.uint64)
        total, ptr = native.C.c_uint64(), native.C.c_void_p()
        native._check(native.lib().mp_job_output_device(job.h, native.C.byref(ptr), native._p64(sizes), native.C.byref(total)),
                      "output_device")
        files = torch.as_tensor(_Bytes(ptr.value, total.value), device="cuda")
    else:
        fno, ofs = native.fastq_index_ptr(c["chunks"], s.host.data_ptr(), s.n, s.il)
        starts = native.chunk_starts_of(fno, ofs, [s.n])
        cnt = job.load_count(s.host.data_ptr(), s.n, k, starts, m3, s.il)
        bounds = job.partition(k, c["scans"], c["threads"], starts, cnt.chunk_first_read, cnt.hist, m3)
        sizes, total = job.output_plan()
        total = job.output_to(s.out.data_ptr(), s.out.numel())
        files = s.out if c["work"] == "ragged" else s.out[:total]  # ragged reads: the whole buffer, zero past the files
    return [cnt.hist.view(np.int64), cnt.chunk_reads.view(np.int64), bounds.view(np.int64), sizes.view(np.int64), files]


def run(s):
    c = s.case
    if c["kind"] == "job":
        return _run_job(s)
    if c["kind"] == "batch":
        res = s.batch.run(c["k"], [native.SampleIn(h.data_ptr(), h.numel(), c["chunks"], c["threads"], o.data_ptr(), o.numel())
                                   for h, o in zip(s.hosts, s.outs)])
        return [np.stack([r["bounds"] for r in res]).astype(np.int64)] + [o[:r["out_total"]] for o, r in zip(s.outs, res)]
    if c["kind"] == "serve":
        tickets = [s.server.submit(h.data_ptr(), h.numel(), s.params, o.data_ptr(), o.numel()) for h, o in zip(s.hosts, s.outs)]
        res = [s.server.result(t) for t in tickets]
        for r in res:
            if r.status:
                raise native.MetapartError(r.error)
        return [np.array([r.bounds for r in res], dtype=np.int64)] + [o[:r.out_total] for o, r in zip(s.outs, res)]
    hi, hi2 = (s.hi.data_ptr(), s.hi2.data_ptr()) if s.hi is not None else (None, None)
    a = (s.lo.data_ptr(), hi, s.id.data_ptr(), s.lo2.data_ptr(), hi2, s.id2.data_ptr(), c["n"])
    stream = torch.cuda.current_stream().cuda_stream
    if c["fixed"]:  # the allocation-free entry point
        rc = native.lib().mp_sort_tuples_noalloc(*(native.C.c_void_p(x) if x else None for x in a[:6]), native.C.c_uint64(a[6]),
                                                 native.C.c_void_p(stream))
        native._check(rc, "mp_sort_tuples_noalloc")
    else:
        native.sort_tuples(s.ctx, *a, stream)
    return [s.lo2, s.id2] + ([s.hi2] if s.hi2 is not None else [])


def work(case):
    if case["kind"] == "sort":
        return {"bytes": 2 * case["n"] * (13 if 2 * case["k"] + 8 > 64 else 12), "flops": 0}
    if case["kind"] == "job":
        length = case["length"]
        if case["work"] == "ragged":
            k = case["k"]
            length = (k - 4 + max(k, length // 2) + max(k, 2 * length // 3) + length) / 4
        reads = case["reads"]
    else:  # read counts log-uniform between lo and hi
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo)
        length, reads = (166.7, mean * case["samples"]) if case["kind"] == "batch" else (150, mean * case["requests"])
    # the FASTQ bytes in, the partition files out
    return {"bytes": 2 * reads * (2 * length + 6 + 7), "flops": 0}


def exact(case, seed):
    """The sorted tuples by torch's stable sort; a job's outputs are whole numbers and bytes with no such value."""
    if case["kind"] != "sort":
        return None
    s = prepare(case, seed)
    lo, order = torch.sort(s.lo ^ (-1 << 63), stable=True)  # unsigned order
    if s.hi is not None:
        hi, second = torch.sort(s.hi[order], stable=True)
        return [lo[second] ^ (-1 << 63), s.id[order[second]], hi]
    return [lo ^ (-1 << 63), s.id[order]]
