"""CRC kernels at the edges of their 16-byte chunks and 512-byte rows.

The buffer CRC and the input-block check both read memory in 16-byte chunks
of the address grid, 32 to a row; sizes and start addresses around a chunk, a
row, a warp's run of rows and one CTA's rows must give the restatement's CRC
(whole numbers: equal, no tolerance)."""
import numpy as np
import pytest

import oracle
from luda_b200 import workloads
from luda_b200.engine import LcError

pytestmark = pytest.mark.gpu

SIZES = [1, 15, 16, 17, 496, 511, 512, 513, 2048 + 16, 16 * 512 * 2 - 1, 16 * 512 * 2 + 33,
         148 * 16 * 512 * 2 + 7, 296 * 16 * 512 * 9 + 500]


@pytest.mark.parametrize("n", SIZES)
def test_buffer_at_every_chunk_phase(engine, n):
    import torch
    b = np.random.default_rng(n).integers(0, 256, n + 16, dtype=np.uint8)
    d = torch.from_numpy(b).cuda()
    torch.cuda.synchronize()
    for off in (range(16) if n < 100000 else (0, 1, 9, 15)):
        want = oracle.crc32c_mask(oracle.crc32c(b[off:off + n].tobytes()))
        assert engine.crc32c(device_ptr=d.data_ptr() + off, n=n) == want, off


@pytest.mark.parametrize("off", [0, 1, 7, 15])
def test_input_check_at_any_table_address(engine, oracle_lib, off):
    import torch
    job = workloads.l0_l1_job(77, n0=2, n1=1, entries_per_table=700, key_space=1 << 20)
    job.materialize(lambda e, o: oracle.build_table(e, o, "oracle"))
    tables = job.input_tables()
    raw = b"".join(f.data for f in tables)
    d = torch.zeros(len(raw) + 64, dtype=torch.uint8, device="cuda")
    d[off:off + len(raw)] = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()
    at = np.cumsum([0] + [len(f.data) for f in tables])
    ptrs = [d.data_ptr() + off + int(a) for a in at[:-1]]
    torch.cuda.synchronize()
    res = engine.compact(job, device_tables=ptrs, verify_checksums=True)
    assert res.file_bytes() == [w[0] for w in oracle.compact(job, "oracle")]
    # one flipped value bit in the first and in a later block is caught
    for pos in (40, 9000, int(at[1]) + 60):
        d[off + pos] ^= 1
        torch.cuda.synchronize()
        with pytest.raises(LcError, match="checksum"):
            engine.compact(job, device_tables=ptrs, verify_checksums=True)
        d[off + pos] ^= 1
        torch.cuda.synchronize()
