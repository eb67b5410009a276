"""Values of uneven length side by side in a block.

Of up to 32 entries at a time, values from 33 bytes to some hundreds are copied
by groups of eight lanes, in steps of 128 bytes that are dealt to the groups
one by one when some value needs more than one.  The cases mix lengths at the
steps' edges, empty values and short ones between them, and lengths drawn over
decades, in blocks assembled whole and in windows.  Output bytes must equal the
restatement's."""
import numpy as np
import pytest

import oracle
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions, internal_key

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(11)
LENGTHS = {
    "edges": [int(128 * k + d) for k in range(1, 5) for d in range(-6, 8)] * 12,
    "empty_between": list(np.where(RNG.random(900) < 0.4, 0, RNG.integers(33, 700, 900))),
    "short_between": list(np.where(RNG.random(900) < 0.6, RNG.integers(0, 40, 900),
                                   RNG.integers(129, 500, 900))),
    "decades": [int(x) for x in np.exp(RNG.normal(5, 1, 1500)).clip(0, 4000)],
    "one_long": [100] * 31 + [1500] + [100] * 40 + [2000, 0, 33, 32, 34, 128, 129],
}


@pytest.mark.parametrize("block", [300, 4096, 5100, 16384])
@pytest.mark.parametrize("name", list(LENGTHS))
def test_uneven_values_match_restatement(engine, oracle_lib, name, block):
    opts = TableOptions(block, 16, 10, 1 << 20)
    lens, files = LENGTHS[name], []
    rng = np.random.default_rng(block)
    for t in range(2):
        part = lens[t::2]
        e = Entries.from_lists(
            [internal_key(b"%09d" % (2 * i + t), 1 + i + 10 ** 6 * t, 1) for i in range(len(part))],
            [rng.bytes(int(n)) for n in part])
        files.append(FileMeta(t, t + 1, e.key(0), e.key(e.n - 1), entries=e))
    job = CompactionJob(0, files, [], 1 << 30, opts, name=name)
    job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))
    res = engine.run(engine.prepare(job))
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    res.release()
