"""Blocks, files and index keys at the edges of the ways they are computed.

A job of at most 8192 entries is partitioned by one kernel (a cluster of 512
threads per 512 entries, up to 8), one of at most 8192 expected blocks has its
blocks laid out by that kernel, larger ones go kernel by kernel.  The cases put
the numbers of entries and blocks at those edges and past them (more blocks
than expected too: values far smaller than the blocks' average), with one
output file or many, cuts at grandparents, restart intervals from 1, and user
keys whose separators are at their limits (0xff runs, prefixes of each other,
zero bytes).  Output bytes must equal the restatement's."""
import numpy as np
import pytest

import oracle
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu


def _user_keys(kind, n, rng):
    if kind == "digits":
        return [b"%08d" % (7 * i) for i in range(n)]
    if kind == "ff":  # 0xff runs and neighbours that differ by one
        alphabet = np.array([0x00, 0x01, 0xfe, 0xff], dtype=np.uint8)
        ks = set()
        while len(ks) < n:
            ks.add(bytes(alphabet[rng.integers(0, 4, int(rng.integers(1, 14)))]))
        return sorted(ks)
    ks, at = set(), 0  # prefixes of each other
    while len(ks) < n:
        base = b"%06d" % at
        for m in range(int(rng.integers(1, 5))):
            ks.add(base + b"a" * m)
        at += 1
    return sorted(ks)[:n]


def _run(engine, n, opts, kind, vmax, gp_every=0):
    rng = np.random.default_rng(n + vmax)
    keys = _user_keys(kind, n, rng)
    cut = max(1, n // 3)
    upper = set(rng.choice(n, cut, replace=False).tolist())
    files = []
    for lv, ids in ((1, [i for i in range(n) if i not in upper]), (0, sorted(upper))):
        if not ids:
            continue
        e = Entries.from_lists([internal_key(keys[i], 1 + i, 1) for i in ids],
                               [rng.bytes(int(rng.integers(0, vmax + 1))) for _ in ids])
        files.append(FileMeta(lv, len(files) + 1, e.key(0), e.key(e.n - 1), entries=e))
    if gp_every:
        for g in range(0, n - gp_every, gp_every):
            files.append(FileMeta(2, 100 + g, internal_key(keys[g], 5, 1),
                                  internal_key(keys[g + gp_every // 2], 5, 1),
                                  file_size=4 * opts.max_file_size))
    job = CompactionJob(0, files, [], 1 << 30, opts, name=kind)
    job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))
    for f in job.files:
        if f.entries is not None:
            assert engine.build_table(f.entries, opts) == f.data
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]


@pytest.mark.parametrize("n", [1, 2, 512, 513, 1025, 4096, 4097, 8191, 8192, 8193, 16384, 40000])
def test_entry_counts(engine, oracle_lib, n):
    _run(engine, n, TableOptions(1024, 16, 10, 1 << 16), "digits", 60)


@pytest.mark.parametrize("n,block", [(9000, 64), (9000, 1), (20000, 64), (20000, 100), (33000, 128),
                                     (9000, 4096), (30000, 300)])
def test_block_counts(engine, oracle_lib, n, block):
    _run(engine, n, TableOptions(block, 4, 10, 1 << 18), "digits", 8)


@pytest.mark.parametrize("kind", ["ff", "prefixes"])
@pytest.mark.parametrize("n,block", [(700, 64), (3000, 256), (9000, 40), (9000, 700)])
def test_index_keys(engine, oracle_lib, kind, n, block):
    _run(engine, n, TableOptions(block, 3, 12, 4096), kind, 12)
    _run(engine, n, TableOptions(block, 1, 0, 4096), kind, 12)


@pytest.mark.parametrize("n", [600, 5000, 9000, 30000])
def test_grandparent_cuts(engine, oracle_lib, n):
    _run(engine, n, TableOptions(512, 16, 10, 8192), "digits", 40, gp_every=max(4, n // 60))


def _long_job(lens, opts, gp_every=0):
    rng = np.random.default_rng(len(lens))
    n = len(lens)
    data = rng.bytes(1 << 20)
    files = []
    for lv in (0, 1):
        ids = range(lv, n, 2)
        e = Entries.from_lists([internal_key(b"%08d" % i, 1 + i, 1) for i in ids],
                               [data[i % 1000:i % 1000 + int(lens[i])] for i in ids])
        files.append(FileMeta(lv, lv + 1, e.key(0), e.key(e.n - 1), entries=e))
    for g in range(0, n - gp_every, gp_every) if gp_every else ():
        files.append(FileMeta(2, 100 + g, internal_key(b"%08d" % g, 5, 1),
                              internal_key(b"%08d" % (g + gp_every // 2), 5, 1),
                              file_size=4 * opts.max_file_size))
    return CompactionJob(0, files, [], 1 << 30, opts).materialize(
        lambda e, o: oracle.build_table(e, o, "oracle"))


@pytest.mark.parametrize("restart", [1, 16, 255])
@pytest.mark.parametrize("kind", ["dense_runs", "big_entries", "plain", "cuts"])
def test_block_starts_of_long_jobs(engine, oracle_lib, kind, restart):
    """More than 131072 survivors: the block starts are searched for in tiles of
    2048 survivors and the 512 after them.  Runs of empty values make blocks
    that reach further, entries of more than 512 KiB leave the 32-bit sums."""
    n, block, gp = 140000, 4096, 0
    lens = np.random.default_rng(7).integers(0, 60, n)
    if kind == "dense_runs":
        block = 8192
        lens = np.where(np.arange(n) // 5000 % 3 < 2, 0, 300)
    elif kind == "big_entries":
        lens[[5, 2047, 2048, 70000, 70001, 139999]] = [600000, 524288, 524270, 530000, 900000, 700000]
    elif kind == "cuts":
        gp = 900
    job = _long_job(lens, TableOptions(block, restart, 10, 1 << 18 if gp else 1 << 22), gp)
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()
