"""Values of many blocks' size: filter and trailer work that grows with the data.

A data block of a 1 MiB value has 512 filter offsets and is written in some 228
windows, so that a job of a few hundred entries has as much of both as one of
a million small entries.  The kernels after the block encoder (k_meta_crc,
k_meta_trailers) take their CTAs from that, not from the number of entries."""
import numpy as np
import pytest

import oracle
from luda_b200.engine import Engine
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu


def _job(n, size, bits, max_file):
    data = np.random.default_rng(size).bytes(size + n)
    files = []
    for lv in (0, 1):
        ids = range(1 - lv, n, 2)
        e = Entries.from_lists([internal_key(b"%08d" % i, 1 + i, 1) for i in ids],
                               [data[i:i + size - 3 * i] for i in ids])
        files.append(FileMeta(lv, lv + 1, e.key(0), e.key(e.n - 1), entries=e))
    job = CompactionJob(0, files, [], 1 << 30, TableOptions(4096, 16, bits, max_file))
    return job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))


@pytest.mark.parametrize("n,size,bits,max_file", [(40, 1 << 20, 10, 2 << 20), (40, 1 << 20, 0, 64 << 20),
                                                  (300, 100000, 16, 32 << 20), (9, 3 << 20, 6, 1 << 20)])
def test_large_values_match_restatement(engine, oracle_lib, n, size, bits, max_file):
    job = _job(n, size, bits, max_file)
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()


def test_meta_phase_is_small_beside_the_encoder(oracle_lib):
    """192 values of 1 MiB in 2 MiB files: 400 KB of filter offsets and 43000
    windows beside 384 MiB that the encoder reads and writes.  Left to one CTA
    and a few hundred threads, a piece or a window after the other (a microsecond
    or more each), they take as long as the encoder; spread over the device,
    some 15 us.  The limit is a third of the encoder's phase."""
    job = _job(192, 1 << 20, 10, 2 << 20)
    best = None
    with Engine(0, phase_timing=True) as eng:
        for _ in range(8):
            res = eng.run(eng.prepare(job))
            ph = dict(res.phase_ms)
            if best is None or ph["encode_meta"] < best["encode_meta"]:
                best = ph
            res.release()
    assert best["encode_meta"] < best["encode_blocks"] / 3, best
