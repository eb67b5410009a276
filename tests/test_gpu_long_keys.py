"""Index keys and filters of many bytes, written beside the data blocks.

An index key of up to 64 bytes is copied by its block's lane, a longer one by a
warp; a filter of more than 1 KiB is built in place; and few blocks are dealt
to warps on different SMs.  The cases put key lengths around the 64 bytes (with
separators shortened to lengths below and above, at every alignment), keys of
many KiB, filters of many KiB, and numbers of blocks from one up.  Output bytes
must equal the restatement's, for a compaction and for the flush encoder."""
import numpy as np
import pytest

import oracle
from luda_b200.engine import Engine
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu


def _job(user_keys, lens, opts):
    data = np.random.default_rng(len(user_keys)).bytes(70000)
    files = []
    for lv in (0, 1):
        ids = range(1 - lv, len(user_keys), 2)
        if not len(ids):
            continue
        e = Entries.from_lists([internal_key(user_keys[i], 1 + i, 1) for i in ids],
                               [data[i % 999:i % 999 + int(lens[i])] for i in ids])
        files.append(FileMeta(lv, lv + 1, e.key(0), e.key(e.n - 1), entries=e))
    job = CompactionJob(0, files, [], 1 << 30, opts)
    return job.materialize(lambda x, o: oracle.build_table(x, o, "oracle"))


def _around(lo, hi, n):
    """Keys of lo..hi bytes that differ early or late (separators of any length)."""
    rng = np.random.default_rng(lo)
    return sorted({b"%05d" % (i // 3) + bytes(rng.integers(97, 99, int(rng.integers(lo, hi + 1)) - 5, dtype=np.uint8))
                   for i in range(n)})


def _long(size, n):
    return [b"%08d" % i + bytes([97 + i % 26]) * (size - 8 - i % 7) for i in range(n)]


KEYS = {
    "around_64": (_around(50, 80, 2500), 40, TableOptions(300, 4, 10, 1 << 20)),
    "around_128": (_around(110, 150, 1500), 40, TableOptions(700, 16, 10, 1 << 20)),
    "around_256": (_around(240, 270, 1000), 40, TableOptions(1024, 16, 10, 1 << 20)),
    "of_5k": (_long(5000, 300), 10, TableOptions(4096, 16, 10, 1 << 20)),
    "of_9k_many_files": (_long(9000, 150), 3000, TableOptions(4096, 2, 0, 1 << 20)),
    "of_60k": (_long(60000, 40), 10, TableOptions(65536, 16, 10, 4 << 20)),
}
FILTERS = {  # entries, value bytes, block size, bits per key
    "one_block": (3000, 5, 1 << 20, 30),
    "few_blocks": (20000, 5, 65536, 20),
    "many_blocks": (60000, 8, 16384, 100),
    "huge_filter": (50000, 0, 1 << 20, 64),
}


@pytest.mark.parametrize("name", list(KEYS))
def test_long_index_keys_match_restatement(engine, oracle_lib, name):
    keys, vlen, opts = KEYS[name]
    job = _job(keys, np.full(len(keys), vlen), opts)
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()
    for f in job.files:
        assert engine.build_table(f.entries, opts) == f.data


@pytest.mark.parametrize("name", list(FILTERS))
def test_large_filters_match_restatement(engine, oracle_lib, name):
    n, vlen, block, bits = FILTERS[name]
    opts = TableOptions(block, 16, bits, 4 << 20)
    job = _job([b"%016d" % (7 * i) for i in range(n)], np.full(n, vlen), opts)
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()
    for f in job.files:
        assert engine.build_table(f.entries, opts) == f.data


def _phases(job):
    best = None
    with Engine(0, phase_timing=True) as eng:
        for _ in range(6):
            res = eng.run(eng.prepare(job))
            if best is None or res.phase_ms["encode_blocks"] < best["encode_blocks"]:
                best = dict(res.phase_ms)
            res.release()
    return best


def test_long_index_keys_are_spread(oracle_lib):
    """1500 keys of 9 KB, a block each: 13 MB of index keys.  Byte by byte by the
    lanes of one CTA (a sector a lane and store) they take 15 ms; copied by warps
    on different SMs some 100 us.  The decode phase of these keys (2.5 ms, an entry
    at a time) is the limit."""
    keys = _long(9000, 1500)
    ph = _phases(_job(keys, np.full(1500, 50), TableOptions(4096, 16, 10, 2 << 20)))
    assert ph["encode_blocks"] < ph["decode"], ph


def test_large_filters_are_spread(oracle_lib):
    """120000 keys at 30 bits in 31 blocks of 64 KiB, 77000 bits to set for each
    filter: by 16 warps of one SM side by side 1.9 ms, fifty times the phase of the
    same keys in 4 KiB blocks; by warps on 31 SMs eight times.  The limit is 20."""
    n = 120000
    keys = [b"%016d" % (7 * i) for i in range(n)]
    ph = [_phases(_job(keys, np.full(n, 5), TableOptions(b, 16, 30, 2 << 20)))["encode_blocks"] for b in (4096, 65536)]
    assert ph[1] < 20 * ph[0], ph
