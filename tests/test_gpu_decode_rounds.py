"""The decode's second pass at the edges of its rounds.

Keys of at most 32 bytes are decoded in registers, a round of 32 entries at a
time, longer ones through shared memory or in the arena; shared prefixes reach
over rounds when a restart run is longer than one.  The cases mix key lengths
around 32 bytes, prefixes that shrink and grow inside and across rounds, runs
of 1 to 255 entries and user keys of 0 to 70 bytes.  Output bytes must equal
the restatement's; the bloom filters check the hashes kept with the keys."""
import numpy as np
import pytest

import oracle
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu


def _keys(kind, n, rng):
    if kind == "short":  # 0 to 24 user-key bytes: every round in registers
        ks = {bytes(rng.integers(97, 100, int(rng.integers(0, 25)), dtype=np.uint8)) for _ in range(n)}
    elif kind == "around_32":  # 20 to 28: rounds change between the two ways
        ks = {b"p" * int(rng.integers(0, 12)) + bytes(rng.integers(97, 123, int(rng.integers(14, 18)),
                                                                   dtype=np.uint8)) for _ in range(n)}
    elif kind == "mixed":  # mostly short, a long key in some rounds
        ks = {b"k%06d" % int(i) + (b"x" * int(rng.integers(20, 64)) if rng.random() < 0.02 else b"")
              for i in rng.integers(0, 10 ** 6, n)}
    elif kind == "deep":  # long shared prefixes of changing length
        ks = {b"%024d" % int(i) for i in rng.integers(0, 5000, n)}
    else:  # zero bytes in and at the end of keys
        ks = {bytes(rng.integers(0, 2, int(rng.integers(1, 14)), dtype=np.uint8)) for _ in range(n)}
    return sorted(ks)


@pytest.mark.parametrize("restart", [1, 2, 16, 33, 64, 255])
@pytest.mark.parametrize("kind", ["short", "around_32", "mixed", "deep", "zeros"])
def test_decode_rounds_match_restatement(engine, oracle_lib, kind, restart):
    rng = np.random.default_rng(restart * 7 + len(kind))
    opts = TableOptions(block_size=4096, restart_interval=restart, bits_per_key=12, max_file_size=1 << 20)
    files, seq = [], 1
    for t in range(3):
        keys = _keys(kind, 3000, rng)
        ik = []
        for k in keys:  # some user keys twice: the tag bytes share prefixes too
            for _ in range(2 if rng.random() < 0.1 else 1):
                ik.append((k, seq))
                seq += 1
        ik.sort(key=lambda x: (x[0], -x[1]))
        e = Entries.from_lists([internal_key(k, s, 1) for k, s in ik],
                               [rng.bytes(int(rng.integers(0, 9))) for _ in ik])
        files.append(FileMeta(1 if t == 0 else 0, t + 1, e.key(0), e.key(e.n - 1), entries=e))
    job = CompactionJob(0, files, [seq // 2], seq, opts, name=kind)
    job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))
    for f in job.files:
        assert engine.build_table(f.entries, opts) == f.data
    res = engine.run(engine.prepare(job, outputs_on_device=2, keep_decoded=True))
    want = [w[0] for w in oracle.compact(job, "oracle")]
    assert res.file_bytes() == want
    # the outputs read back from their decoded form
    outs = [FileMeta(1, 10 + i, f.smallest, f.largest, data=bytes(f.data), file_size=len(f.data))
            for i, f in enumerate(res.files)]
    again = CompactionJob(1, outs, [], seq, opts)
    got = engine.run(engine.prepare(again, [res.device_ptr + o for o in res.file_offsets],
                                    decoded=[f.decoded for f in res.files]))
    assert got.file_bytes() == [w[0] for w in oracle.compact(again, "oracle")]
    got.release()
    res.release()
