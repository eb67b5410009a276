"""Data blocks around and beyond the block encoder's stage.

A block of up to 5056 bytes is assembled whole by one warp; a wider one in
windows of 4608 bytes by several, its CRC put together from theirs.  The cases
set block sizes at those edges (every length around them, at every 16-byte
phase the blocks before them leave), blocks of thousands of entries (the
window's first entry is found from prefix sums; restart arrays longer than a
window), empty values, and values many windows long.  Output bytes must equal
the restatement's, for a compaction, from its decoded form, and for the flush
encoder."""
import numpy as np
import pytest

import oracle
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu


def _entries(lens, seq0, klen, seed):
    rng = np.random.default_rng(seed)
    keys = [internal_key(b"%0*d" % (klen, 3 * i + seq0 % 3), seq0 + i, 1) for i in range(len(lens))]
    return Entries.from_lists(keys, [rng.bytes(int(n)) for n in lens])


def _job(lens, opts, klen=12, seed=1):
    """Two level-0 tables and a level-1 table whose keys interleave."""
    files = []
    for t in range(3):
        e = _entries(lens[t::3], 1 + 100000 * t, klen, seed + t)
        files.append(FileMeta(1 if t == 0 else 0, t + 1, e.key(0), e.key(e.n - 1), entries=e))
    job = CompactionJob(0, files, [], 1 << 30, opts, name="wide")
    return job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))


EDGES = list(range(4990, 5080)) + list(range(4560, 4660)) + list(range(9160, 9250))
RNG = np.random.default_rng(5)
CASES = {
    "edges": (EDGES, TableOptions(block_size=1024, restart_interval=16, bits_per_key=10)),
    "long": ([70000, 3, 4608 * 4 - 20, 0, 16384, 65535, 131072, 9, 200000, 4096, 5000, 30000],
             TableOptions(block_size=4096, restart_interval=2, bits_per_key=0)),
    "many_small": (RNG.integers(0, 6, 30000), TableOptions(65536, 16, 10, 1 << 20)),
    "every_restart": (RNG.integers(0, 40, 12000), TableOptions(65536, 1, 10, 1 << 20)),
    "odd_interval": (RNG.integers(0, 300, 6000), TableOptions(32768, 11, 16, 1 << 20)),
    "long_interval": (RNG.integers(20, 140, 6000), TableOptions(16384, 255, 10, 1 << 20)),
    "mixed": (np.where(RNG.random(2000) < 0.05, 6000, RNG.integers(0, 900, 2000)),
              TableOptions(8192, 16, 10, 1 << 20)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_wide_blocks_match_restatement(engine, oracle_lib, name):
    lens, opts = CASES[name]
    job = _job(list(lens), opts)
    for f in job.files:
        assert engine.build_table(f.entries, opts) == f.data
    want = oracle.compact(job, "oracle")
    res = engine.run(engine.prepare(job, outputs_on_device=2, keep_decoded=True))
    assert res.file_bytes() == [w[0] for w in want]
    # a second job reads the outputs from their decoded form (value places)
    files = [FileMeta(1, 10 + i, f.smallest, f.largest, data=bytes(f.data), file_size=len(f.data))
             for i, f in enumerate(res.files)]
    second = CompactionJob(1, files, [], 1 << 30, opts)
    ptrs = [res.device_ptr + o for o in res.file_offsets]
    got = engine.run(engine.prepare(second, ptrs, decoded=[f.decoded for f in res.files]))
    assert got.decoded_inputs == len(files)
    assert got.file_bytes() == [w[0] for w in oracle.compact(second, "oracle")]
    got.release()
    res.release()
