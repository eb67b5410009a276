"""Blocks of many more entries than a job's average one.

The block starts of long jobs (more than 131072 survivors, at most 256 entries a
block on average) are searched for in tiles of 2048 survivors and the 512 after
them.  Stretches of empty values make blocks that reach past those: their ends
are found span by span.  The cases put such stretches at the tiles' edges, with
blocks of a few to many spans, cut at grandparents, between entries of more
than 512 KiB, at the job's end.  Output bytes must equal the restatement's."""
import numpy as np
import pytest

import oracle
from luda_b200.engine import Engine
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu


def _entries(lens):
    n = len(lens)
    ids = np.arange(n)
    digits = ((ids[:, None] // 10 ** np.arange(15, -1, -1)) % 10 + 48).astype(np.uint8)
    tags = ((ids + 1) << 8 | 1).astype("<u8").view(np.uint8).reshape(n, 8)
    voffs = np.zeros(n + 1, np.uint64)
    voffs[1:] = np.cumsum(lens)
    vals = np.random.default_rng(1).integers(0, 256, int(voffs[-1]), dtype=np.uint8)
    return Entries(np.concatenate([digits, tags], 1).reshape(-1), np.arange(n + 1, dtype=np.uint64) * 24,
                   vals, voffs)


def _job(lens, opts, gp=()):
    e = _entries(lens)
    files = [FileMeta(0, 1, e.key(0), e.key(e.n - 1), entries=e)]
    for g in gp:
        files.append(FileMeta(2, 100 + g, internal_key(b"%016d" % g, 5, 1), internal_key(b"%016d" % (g + 9), 5, 1),
                              file_size=4 * opts.max_file_size))
    job = CompactionJob(0, files, [], 1 << 30, opts)
    return job.materialize(lambda x, o: oracle.build_table(x, o, "oracle"))


def _skew(n, period, empty, size, block):
    """`empty` of each `period` values are empty; checked to lie on the searched path."""
    lens = np.where(np.arange(n) % period < empty, 0, size)
    assert n > 131072 and block <= 256 * (12 + lens.mean())  # an entry's least bytes
    return lens


def _cases():
    n = 150000
    yield "half_span", _skew(n, 5000, 4000, 700, 16384), TableOptions(16384, 16, 10, 1 << 21), ()
    yield "spans", _skew(n, 30000, 27000, 2600, 65000), TableOptions(65000, 16, 10, 1 << 22), ()
    yield "many_spans", _skew(n, 50000, 47000, 17000, 262144), TableOptions(262144, 16, 10, 1 << 23), ()
    yield "every_restart", _skew(n, 7000, 6000, 900, 32768), TableOptions(32768, 1, 0, 1 << 21), ()
    yield "odd_restart", _skew(n, 7001, 5999, 1000, 32768), TableOptions(32768, 11, 10, 1 << 21), ()
    yield "long_restart", _skew(n, 7001, 5999, 1000, 32768), TableOptions(32768, 255, 10, 1 << 21), ()
    yield ("cuts", _skew(n, 30000, 27000, 1400, 32768), TableOptions(32768, 16, 10, 1 << 18),
           tuple(range(100, n - 100, 1700)))
    lens = _skew(n, 30000, 27000, 1400, 32768)
    lens[[0, 2047, 2048, 2559, 2560, 4607, 4608, 26999, 60000, 60001, n - 1]] = [
        600000, 524288, 524270, 530000, 700000, 524256, 524280, 900000, 600000, 524289, 600000]
    yield "big_entries", lens, TableOptions(32768, 16, 10, 1 << 21), ()
    lens = _skew(n, 30000, 27000, 1400, 32768)
    lens[-20000:] = 0
    yield "to_the_end", lens, TableOptions(32768, 16, 10, 1 << 21), ()


CASES = {name: rest for name, *rest in _cases()}


@pytest.mark.parametrize("name", list(CASES))
def test_long_blocks_match_restatement(engine, oracle_lib, name):
    lens, opts, gp = CASES[name]
    job = _job(lens, opts, gp)
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()
    if not gp:
        assert engine.build_table(job.files[0].entries, opts) == job.files[0].data


def test_long_blocks_cost_no_walk(oracle_lib):
    """400000 entries in 32 KiB blocks, nine tenths of them empty values that make
    blocks of 2730.  Walked entry by entry, a dependent load each, the block ends
    took 17 times as long as the job's decode and encoder phases together; found
    by searches they take about as long as these.  The limit is five times."""
    lens, opts = _skew(400000, 20000, 18000, 1400, 32768), TableOptions(32768, 16, 10, 8 << 20)
    e = _entries(lens)
    got = []
    with Engine(0, phase_timing=True) as eng:
        job = CompactionJob(0, [FileMeta(0, 1, e.key(0), e.key(e.n - 1), data=eng.build_table(e, opts))], [], 1 << 30,
                            opts)
        for _ in range(6):
            res = eng.run(eng.prepare(job))
            got.append(res.phase_ms["partition"] / (res.phase_ms["decode"] + res.phase_ms["encode_blocks"]))
            res.release()
    assert min(got) < 5, got
