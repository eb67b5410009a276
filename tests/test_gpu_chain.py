"""The block chain when its chunk tables do not fit shared memory.

The chain of block starts is followed chunk by chunk (4096 survivors, or 1024
in small jobs of short blocks), through tables as wide as the longest block.
With small values a block has hundreds of entries: a few dozen chunks then
need more than the 44 KiB that the tables are staged in, although they are
fewer than one group of chunks (64).  Every case states its chunk and is
checked to lie there, by a model of the block builder over its keys and
values.  A job of another shape runs first, so that the scratch memory holds
its remains.  Output bytes must equal the restatement's."""
import numpy as np
import pytest

import oracle
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

SMEM_WORDS, GROUP = 11 * 1024, 64


def _varint_len(x):
    return 1 if x < 128 else 2 if x < 1 << 14 else 3


def longest_block(keys, lens, opts):
    """Entries of the longest data block (BlockBuilder's size estimate)."""
    most = n = size = restarts = run = 0
    prev = b""
    for k, v in zip(keys, lens):
        shared = 0
        if n and run < opts.restart_interval:
            m = min(len(k), len(prev))
            while shared < m and k[shared] == prev[shared]:
                shared += 1
        else:
            restarts, run = restarts + 1, 0
        rest = len(k) - shared
        size += _varint_len(shared) + _varint_len(rest) + _varint_len(int(v)) + rest + int(v)
        n, run, prev = n + 1, run + 1, k
        if size + 4 * restarts + 4 >= opts.block_size:
            most, n, size, restarts = max(most, n), 0, 0, 0
    return max(most, n)


def user_key(i, klen):
    return b"%0*d" % (klen - 8, i)


def value_lens(n, lo, hi, runs=()):
    """n lengths in [lo, hi); `runs`: (first, count) of empty values."""
    v = np.random.default_rng(n + hi).integers(lo, hi, n)
    for a, c in runs:
        v[a:a + c] = 0
    return v


# entries, internal key bytes, value lengths, block size, restart interval, chunk
COMPACTIONS = {
    "16k_blocks": (100000, 16, (0, 13), 16384, 16, 4096),
    "32k_blocks": (60000, 16, (0, 41), 32768, 16, 4096),
    "64k_blocks": (30000, 16, (0, 33), 65536, 16, 4096),
    "odd_restarts": (90000, 24, (0, 7), 16384, 11, 4096),
    "8k_blocks_most_chunks": (131000, 16, (0, 3), 8192, 16, 4096),
    "short_chunks": (30000, 16, (60, 140, ((11000, 900),)), 8192, 16, 1024),
    "short_chunks_odd": (32000, 16, (80, 90, ((100, 420), (31400, 600))), 5003, 64, 1024),
}
FLUSHES = {
    "default_blocks": (250000, 24, (0, 3), 4096, 16),
    "16k_blocks": (200000, 16, (0, 13), 16384, 16),
    "64k_blocks": (50000, 16, (0, 9), 65536, 64),
}


def reaches(keys, lens, opts, chunk):
    w = longest_block(keys, lens, opts)
    chunks = -(-len(keys) // chunk)
    assert w <= chunk and chunks <= GROUP and chunks * w > SMEM_WORDS, (w, chunks)


def compaction(name):
    n, klen, vals, block, restart, chunk = COMPACTIONS[name]
    opts = TableOptions(block, restart, 10, 1 << 21)
    lens = value_lens(n, *vals)
    keys = [internal_key(user_key(i, klen), 1 + i, 1) for i in range(n)]
    reaches(keys, lens, opts, chunk)
    data = np.random.default_rng(n).bytes(1 << 16)
    files = []
    for lv in (0, 1):  # odd ids over even ones
        ids = range(1 - lv, n, 2)
        e = Entries.from_lists([keys[i] for i in ids], [data[i % 999:i % 999 + int(lens[i])] for i in ids])
        files.append(FileMeta(lv, lv + 1, e.key(0), e.key(e.n - 1), entries=e))
    # the host's rule for the short chunks, from the input's bytes
    per = sum(len(k) for k in keys) / n + float(np.mean(lens))
    assert (chunk == 1024) == (n < 148 * 1024 and block < 256 * 0.75 * per)
    return CompactionJob(0, files, [], 1 << 30, opts, name=name)


def flush(name):
    n, klen, vals, block, restart = FLUSHES[name]
    opts = TableOptions(block, restart, 10, 1 << 21)
    lens = value_lens(n, *vals)
    keys = [internal_key(user_key(i, klen), 1 + i, 1) for i in range(n)]
    reaches(keys, lens, opts, 4096)
    data = np.random.default_rng(n).bytes(1 << 16)
    return Entries.from_lists(keys, [data[i % 999:i % 999 + int(v)] for i, v in enumerate(lens)]), opts


@pytest.fixture(scope="module")
def other_job(engine, oracle_lib):
    """Leaves the remains of a larger job of short blocks in the scratch memory."""
    n = 300000
    e = Entries.from_lists([internal_key(user_key(7 * i, 20), n + i, 1) for i in range(n)],
                           [b"v" * (i % 90) for i in range(n)])
    opts = TableOptions(1024, 16, 10, 1 << 20)
    f = FileMeta(0, 1, e.key(0), e.key(e.n - 1), entries=e)
    job = CompactionJob(0, [f], [], 1 << 30, opts)
    job.materialize(lambda x, o: engine.build_table(x, o))

    def run():
        engine.run(engine.prepare(job)).release()
    return run


@pytest.mark.parametrize("name", list(COMPACTIONS))
def test_cases_reach_the_unstaged_tables(name):
    compaction(name)


@pytest.mark.parametrize("name", list(FLUSHES))
def test_flushes_reach_the_unstaged_tables(name):
    flush(name)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(COMPACTIONS))
def test_compaction_matches_restatement(engine, oracle_lib, other_job, name):
    job = compaction(name)
    job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))
    want = [w[0] for w in oracle.compact(job, "oracle")]
    other_job()
    for _ in range(3):  # launched one by one, captured, replayed
        res = engine.run(engine.prepare(job))
        assert res.file_bytes() == want
        res.release()


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(FLUSHES))
def test_flush_matches_restatement(engine, oracle_lib, other_job, name):
    entries, opts = flush(name)
    want = oracle.build_table(entries, opts, "oracle")
    other_job()
    assert engine.build_table(entries, opts) == want


# A block of more survivors than a short chunk among blocks of some 60: the job
# goes by long chunks, and is not walked block by block.
def stretch(count):
    n, opts = 60000, TableOptions(16384, 16, 10, 1 << 21)
    lens = value_lens(n, 240, 260, ((20000, count),))
    keys = [internal_key(user_key(i, 16), 1 + i, 1) for i in range(n)]
    e = Entries.from_lists(keys, [b"v" * int(v) for v in lens])
    f = FileMeta(0, 1, e.key(0), e.key(n - 1), entries=e)
    job = CompactionJob(0, [f], [], 1 << 30, opts)
    job.materialize(lambda x, o: oracle.build_table(x, o, "oracle"))
    return job, longest_block(keys, lens, opts)


@pytest.mark.gpu
def test_one_long_block_costs_no_serial_walk(oracle_lib):
    """Of some 940 blocks.  Walked one after the other by a thread (a dependent
    load of device memory each, half a microsecond or more) they take 500 us,
    where the whole partition phase of the job without the stretch takes about
    100: four times that is the limit."""
    from luda_b200.engine import Engine
    ms = []
    with Engine(0, phase_timing=True) as eng:
        for count in (0, 3000):
            job, longest = stretch(count)
            assert longest <= 256 if not count else 1024 < longest <= 4096
            got = []
            for _ in range(8):
                res = eng.run(eng.prepare(job))
                got.append(res.phase_ms["partition"])
                files = res.file_bytes()
                res.release()
            assert files == [w[0] for w in oracle.compact(job, "oracle")]
            ms.append(min(got))
    assert ms[1] < 4 * ms[0], ms
