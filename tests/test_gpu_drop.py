"""The drop rule and the gather of the survivors: tiles of one position a thread
(128) in small jobs, of four (512) in large ones, and the comparison of user
keys behind their prefixes."""
import numpy as np
import pytest

import oracle
from luda_b200.engine import Engine
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu

SMALL_MAX = 148 * 8 * 512  # positions (rounded up to a power of two) from which a thread takes four


def _job(keys, per_key, tomb, snapshots=(), deeper=0, opts=None):
    """Sorted `keys`, `per_key` versions of each over two runs, a share of them
    deletions; `deeper` files two levels below, each over a stretch of keys."""
    rng = np.random.default_rng(len(keys))
    n = len(keys) * per_key
    seqs = 1 + rng.permutation(n).reshape(len(keys), per_key)
    dead = rng.random((len(keys), per_key)) < tomb
    runs = [], []  # (level 0, level 1)
    for i, k in enumerate(keys):
        order = np.argsort(-seqs[i])
        for j in order:
            runs[(i + j) % 2].append((internal_key(k, int(seqs[i, j]), 0 if dead[i, j] else 1),
                                      b"" if dead[i, j] else b"v%d" % seqs[i, j]))
    files = []
    for lv in (0, 1):
        if not runs[lv]:
            continue
        e = Entries.from_lists(*map(list, zip(*runs[lv])))
        files.append(FileMeta(lv, lv + 1, e.key(0), e.key(e.n - 1), entries=e))
    step = max(2, len(keys) // deeper) if deeper else 0
    for d in range(deeper):
        a, b = d * step, min(d * step + step // 2, len(keys) - 1)
        if a < b:
            files.append(FileMeta(2, 100 + d, internal_key(keys[a], 1, 1), internal_key(keys[b], 1, 1), 3 << 20))
    job = CompactionJob(0, files, list(snapshots), 1 << 30, opts or TableOptions(4096, 16, 10, 2 << 20))
    return job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))


def _check(engine, job):
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 255, 257, 511, 512, 513, 1025, 1537])
@pytest.mark.parametrize("per_key,tomb,deeper", [(1, 1.0, 5), (3, 0.3, 0), (2, 0.5, 9)])
def test_tile_edges(engine, oracle_lib, n, per_key, tomb, deeper):
    keys = [b"user%010d" % (3 * i) for i in range((n + per_key - 1) // per_key)]
    _check(engine, _job(keys, per_key, tomb, [n // 2] if per_key == 2 else [], deeper))


@pytest.mark.parametrize("past", [0, 1])
def test_both_tiles_at_the_limit(engine, oracle_lib, past):
    """The largest job of short tiles and the smallest of long ones (the number of
    positions is rounded up to a power of two)."""
    n = 1 << (SMALL_MAX.bit_length() - 1)
    assert n < SMALL_MAX <= 2 * n
    keys = [b"%07d" % i for i in range((n + past + 1) // 2)]
    job = _job(keys, 2, 0.1, [n // 3], 6, TableOptions(4096, 16, 0, 2 << 20))
    if not past:
        assert sum(f.entries.n for f in job.files if f.entries) == n
    _check(engine, job)


def test_nested_keys(engine, oracle_lib):
    """Keys that are heads of one another, several versions each."""
    for byte in (b"\xff", b"a", b"\0"):
        _check(engine, _job([byte * k for k in range(1, 400, 3)], 3, 0.3, [], 4))


@pytest.mark.parametrize("skip", [0, 5])
def test_differing_byte_behind_the_prefix(engine, oracle_lib, skip):
    """Neighbours that differ first at every place from the prefix's last byte to
    40 bytes on, with both lengths: word by word from any alignment."""
    keys = set()
    for at in range(7, 48):
        for c in b"\x01\x7f\x80\xff":
            for more in range(5):
                keys.add(b"p" * (skip + at) + bytes([c]) + b"z" * more)
        keys.add(b"p" * (skip + at))
    _check(engine, _job(sorted(keys), 2, 0.2, [], 6))



def test_long_equal_keys(oracle_lib):
    """Two versions of each of four keys of 5 KB in two runs.  Compared byte by byte
    the merge's rounds (a tile's cuts, a thread's place in it, the merge itself)
    take 1.5 times the decode phase of these keys, word by word two thirds."""
    job = _job([b"k%d" % i * 2500 for i in range(4)], 2, 0.0)
    with Engine(0, phase_timing=True) as eng:
        res = [eng.run(eng.prepare(job)) for _ in range(6)]
        assert min(r.phase_ms["merge"] for r in res) < min(r.phase_ms["decode"] for r in res)


def _drop_us(job):
    best = None
    with Engine(0, phase_timing=True) as eng:
        for _ in range(6):
            res = eng.run(eng.prepare(job))
            us = 1e3 * res.phase_ms["drop"]
            best = us if best is None else min(best, us)
            res.release()
    return best


def test_deletions_of_a_small_job_side_by_side(oracle_lib):
    """Deletions are looked up in the files below, long comparisons where keys
    share 200 bytes.  120 of them in one warp, a strip of 32 after the other, take
    four times as long as 30; in four warps no longer.  The limit is twice."""
    us = []
    for n in (30, 120):
        keys = [b"k" * 200 + b"%06d" % (37 * i) for i in range(n)]
        us.append(_drop_us(_job(keys, 1, 1.0, [], 7)))
    assert us[1] < 2 * us[0], us
