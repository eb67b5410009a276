"""Measured cases: the work a user of the engine has it do.

Each case is one call (or one batch of calls) into ``luda_b200.engine.Engine``:
a compaction (the drop-in for ``DBImpl::DoCompactionWork``) with its tables in
host memory or already in device memory, a batch of compactions, a memtable
flush, or a file checksum.  ``prepare`` makes what the host program holds
before the call (tables, their addresses, the descriptor); ``run`` makes the
call and returns the output bytes, the files' sizes and their boundary keys.

All inputs are synthetic: random values, keys of the shapes the benchmark's
workloads use (``%016d`` decimals, big-endian u64, 24-byte hashed, 8-64-byte
strings with shared prefixes).  One engine serves the whole process, as in a
database server.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from luda_b200.engine import Engine
from luda_b200.job import CompactionJob, Entries, FileMeta, TableOptions

KiB, MiB = 1 << 10, 1 << 20
DELETION, VALUE = 0, 1
KEY16_SPACE = 1 << 26  # ids behind the 16-byte decimal keys
VAR_SPACE = 1 << 24    # ids behind the 8-64-byte keys

_shared_engine = None


def _engine() -> Engine:
    global _shared_engine
    if _shared_engine is None:
        _shared_engine = Engine(0)
    return _shared_engine


# --------------------------------------------------------------------------
# the cases

# What every compaction case may set, and LevelDB's usual values for it.
# "upper" tables of level L over "lower" tables of level L+1, "entries" each.
_COMPACT = dict(kind="compact", level=0, upper=2, lower=2, entries=20000, klen=16, vlen=100,
                vdist="fixed", rewrite=0.10, tomb=0.02, snapshot=False, grandparents=0,
                block=4096, restart=16, bits=10, max_file=2 * MiB, where="device",
                verify=False, chained=False)


def _compact(name=None, **kw):
    c = dict(_COMPACT, **kw)
    if name:
        c = dict(name=name, **c)
    return c


def listed():
    return [
        # A small database's level-0 compaction (about 100 KB): what a job costs when
        # only launches, host synchronisations and latency count.
        _compact("l0_tiny", upper=2, lower=0, entries=400),
        # A full 4 MiB memtable written to a level-0 table (BuildTable), host to host.
        dict(name="flush_4m", kind="flush", entries=35200, klen=16, vlen=100, vdist="fixed",
             tomb=0.02, block=4096, restart=16, bits=10),
        # The benchmark's plain L0->L1 compaction through host buffers: one
        # DoCompactionWork call of an unmodified LevelDB host.
        _compact("l0_l1_host", where="host"),
        # The same shape with paranoid_checks: every input block's checksum verified.
        _compact("l0_l1_paranoid", verify=True),
        # The served loop's chained job: new level-0 tables over level-1 tables that an
        # earlier job left on the device decoded; outputs kept on the device, decoded,
        # and copied to the host to be written.
        _compact("l0_l1_chained", upper=4, lower=4, entries=17600, chained=True),
        # The benchmark's L1->L2 compaction at size (about 66 MiB): 8-64-byte keys,
        # lognormal values, snapshots, deletions, grandparents below half the range.
        _compact("l1_l2_varlen", level=1, upper=1, lower=32, entries=8100, klen=0, vlen=128,
                 vdist="lognormal", rewrite=0.3, tomb=0.05, snapshot=True, grandparents=160),
        # The benchmark's batched mode at half its job count: uneven level-0 jobs in one
        # call, 1-64 MiB each, as many databases share one card.
        dict(name="batch_uneven", kind="batch", jobs=32, lo_kib=1024, hi_kib=65536, shapes=7,
             vlen=100),
        # Larger blocks (16 KiB) without filters, as a scan-heavy store sets them.
        _compact("blocks_16k", level=1, upper=1, lower=16, entries=46000, klen=24, vlen=150,
                 vdist="lognormal", block=16384, bits=0, max_file=8 * MiB, rewrite=0.2),
        # Values larger than a block (documents, serialised objects): 4-64 KiB each.
        _compact("big_values", level=1, upper=1, lower=15, entries=850, klen=24, vlen=16384,
                 vdist="loguniform", max_file=32 * MiB, rewrite=0.2, snapshot=True),
        # The benchmark's headline: 1 GiB of 8-byte keys and 1 KiB values, L2->L3.
        _compact("large_1k_values", level=2, upper=1, lower=15, entries=64340, klen=8, vlen=1024,
                 tomb=0.01, snapshot=True, max_file=64 * MiB),
        # Its entry-heavy run: 24-byte keys and 32-byte values (half of the 1 GiB).
        _compact("large_32b_values", level=2, upper=1, lower=15, entries=500000, klen=24, vlen=32,
                 tomb=0.01, snapshot=True, max_file=64 * MiB),
        # The checksum of a 64 MiB table file in device memory (a backup or scrub pass).
        dict(name="crc_file", kind="crc", size=64 * MiB, offset=0),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """Another case of the ranges the listed ones stand for."""
    what = rng.choice(["l0", "l0", "deep", "deep", "large", "chained", "batch", "flush", "crc"])
    opts = dict(block=rng.choice([4096, 4096, 4096, 1024, 8192, 16384, 32768, 65536]),
                restart=rng.choice([16, 16, 16, 1, 8, 11, 64]),
                bits=rng.choice([10, 10, 10, 0, 6, 16]))
    if what == "crc":
        return dict(kind="crc", size=_log_int(rng, 4 * KiB, 256 * MiB), offset=rng.randrange(16))
    if what == "flush":
        vlen = _log_int(rng, 1, 4096)
        return dict(kind="flush", entries=max(1, _log_int(rng, 64 * KiB, 64 * MiB) // (vlen + 24)),
                    klen=rng.choice([16, 8, 24, 0]), vlen=vlen,
                    vdist=rng.choice(["fixed", "lognormal"]), tomb=rng.choice([0.0, 0.02, 0.2]),
                    **opts)
    if what == "batch":
        hi = _log_int(rng, 512, 32768)
        return dict(kind="batch", jobs=rng.randint(2, 40), lo_kib=max(64, hi // 64), hi_kib=hi,
                    shapes=rng.randrange(1000), vlen=_log_int(rng, 8, 1000))
    upper = rng.randint(1, 8) if what in ("l0", "chained") else rng.randint(1, 2)
    lower = rng.randint(0 if what == "l0" else 1, 12)
    vdist = rng.choice(["fixed", "lognormal"])
    if what == "large":
        vlen, total = _log_int(rng, 16, 1500), _log_int(rng, 64 * MiB, 512 * MiB)
    elif what == "deep":
        vlen, total = _log_int(rng, 8, 4096), _log_int(rng, 2 * MiB, 128 * MiB)
        if rng.random() < 0.2:
            vlen, vdist = _log_int(rng, 4096, 32768), "loguniform"
    else:
        vlen, total = _log_int(rng, 1, 1024), _log_int(rng, 64 * KiB, 32 * MiB)
    entries = max(16, total // (upper + lower) // (vlen + 30))
    entries = min(entries, 4_000_000 // (upper + lower))
    level = 0 if what in ("l0", "chained") else rng.randint(1, 3)
    klen = 16 if level == 0 else rng.choice([0, 8, 24, 24])
    if klen == 0:
        entries = min(entries, VAR_SPACE // 40 // (upper + lower))
    return _compact(level=level, upper=upper, lower=lower, entries=entries, klen=klen, vlen=vlen,
                    vdist=vdist, rewrite=rng.choice([0.0, 0.1, 0.5]),
                    tomb=rng.choice([0.0, 0.02, 0.1]), snapshot=rng.random() < 0.5,
                    grandparents=rng.choice([0, 0, 12, 160]) if level else 0,
                    max_file=rng.choice([2, 2, 8, 64]) * MiB,
                    where="host" if what == "l0" and rng.random() < 0.4 else "device",
                    verify=rng.random() < 0.25, chained=what == "chained", **opts)


# --------------------------------------------------------------------------
# inputs

def _rand(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _perm(g, n):
    return torch.randperm(n, generator=g, device="cuda")


def _zipf(g, n, space=VAR_SPACE, s=0.99):
    a = 1.0 - s
    k = (1.0 + _rand(g, n) * (space ** a - 1.0)) ** (1.0 / a)
    return ((k.long().clamp(1, space) - 1) * 0x9E3779B1) % space


def _distinct(g, n, klen):
    """n distinct ids (a few fewer when the space is crowded), ascending."""
    if n == 0:
        return torch.zeros(0, dtype=torch.long, device="cuda")
    ids = torch.zeros(0, dtype=torch.long, device="cuda")
    for _ in range(8):
        m = 2 * (n - len(ids)) + 64
        if klen == 0:
            more = _zipf(g, 2 * m)
        else:
            space = KEY16_SPACE if klen == 16 else 1 << 62
            more = torch.randint(0, space, (m,), generator=g, device="cuda")
        ids = torch.unique(torch.cat([ids, more]))
        if len(ids) >= n:
            break
    if len(ids) > n:
        ids = torch.sort(ids[_perm(g, len(ids))[:n]]).values
    return ids


def _mix(x):
    """splitmix64's output function on int64 (logical shifts)."""
    def shr(v, s):
        return (v >> s) & ((1 << (64 - s)) - 1)
    z = x - 0x61C8864680B583EB
    z = (z ^ shr(z, 30)) * -0x40A7B892E31B1A47
    z = (z ^ shr(z, 27)) * -0x6B2FB644ECCEEE15
    return z ^ shr(z, 31)


def _be_bytes(v, count=8):
    sh = torch.arange(8 * (count - 1), -1, -8, device="cuda")
    return ((v[:, None] >> sh) & 255).to(torch.uint8)


def _hex(v, digits):
    sh = torch.arange(4 * (digits - 1), -1, -4, device="cuda")
    d = (v[:, None] >> sh) & 15
    return (d + 48 + (d > 9) * 39).to(torch.uint8)


def _user_keys(ids, klen):
    """Key bytes (n, width) and lengths for each id."""
    n = len(ids)
    if klen == 16:
        p10 = torch.tensor([10 ** i for i in range(15, -1, -1)], device="cuda")
        m = ((ids[:, None] // p10) % 10 + 48).to(torch.uint8)
    elif klen == 8:
        m = _be_bytes(ids)
    elif klen:
        tails = [_be_bytes(ids)]
        h = ids
        while sum(t.shape[1] for t in tails) < klen:
            h = _mix(h)
            tails.append(_be_bytes(h))
        m = torch.cat(tails, 1)[:, :klen]
    else:
        # 8-64 bytes, most with one of 32 prefixes: "t07:" + 8 hex digits + filler
        h = _mix(ids)
        lens = 8 + (h & 0xFFFF) % 57
        grp = (h >> 20) & 31
        name, fill = _hex(ids, 8), _hex(_mix(h), 16).repeat(1, 4)
        pre = torch.stack([torch.full_like(grp, 116), grp // 10 + 48, grp % 10 + 48,
                           torch.full_like(grp, 58)], 1).to(torch.uint8)
        m = torch.where((lens >= 12)[:, None], torch.cat([pre, name, fill[:, :52]], 1),
                        torch.cat([name, fill[:, :56]], 1))
        m = torch.where(torch.arange(64, device="cuda") < lens[:, None], m, 0)
        return m, lens
    return m, torch.full((n,), m.shape[1], device="cuda")


def _key_order(m):
    """Positions in byte order of the zero-padded keys (ASCII, no zero bytes)."""
    order = torch.arange(len(m), device="cuda")
    sh = torch.arange(56, -1, -8, device="cuda")
    words = (m.reshape(len(m), -1, 8).long() << sh).sum(2)
    for w in range(words.shape[1] - 1, -1, -1):
        order = order[torch.sort(words[order, w], stable=True).indices]
    return order


def _value_lens(g, n, mean, dist):
    if dist == "fixed":
        return torch.full((n,), mean, device="cuda")
    if dist == "lognormal":  # median `mean`, clipped as the at-size workload clips
        v = torch.exp(torch.randn(n, generator=g, device="cuda", dtype=torch.float64)) * mean
        return v.round().long().clamp(0, 32 * mean)
    lo, hi = math.log(mean / 4), math.log(mean * 4)  # "loguniform" around `mean`
    return torch.exp(lo + _rand(g, n) * (hi - lo)).long()


def _entries(g, ids, seqs, c) -> Entries:
    """Sorted internal keys and random values of the given ids, on the host."""
    m, lens = _user_keys(ids, c["klen"])
    if c["klen"] == 0:
        order = _key_order(m)
        m, lens, seqs = m[order], lens[order], seqs[order]
    n, width = m.shape
    dead = _rand(g, n) < c["tomb"]
    tag = (seqs << 8) | torch.where(dead, DELETION, VALUE)
    tag_bytes = _be_bytes(tag).flip(1)
    if c["klen"]:
        keys = torch.cat([m, tag_bytes], 1).reshape(-1)
    else:
        cols = torch.arange(width + 8, device="cuda")
        at = (cols - lens[:, None]).clamp(0, 7)
        full = torch.cat([m, m[:, :8]], 1)
        full = torch.where(cols < lens[:, None], full, torch.gather(tag_bytes, 1, at))
        keys = full[cols < lens[:, None] + 8]
    koffs = np.zeros(n + 1, np.uint64)
    koffs[1:] = torch.cumsum(lens + 8, 0).cpu().numpy()
    vlens = torch.where(dead, 0, _value_lens(g, n, c["vlen"], c["vdist"]))
    voffs = np.zeros(n + 1, np.uint64)
    voffs[1:] = torch.cumsum(vlens, 0).cpu().numpy()
    words = torch.randint(-(1 << 62), 1 << 62, (int(voffs[-1]) // 8 + 1,), generator=g,
                          device="cuda")
    vals = words.view(torch.uint8)[:int(voffs[-1])]
    return Entries(keys.cpu().numpy(), koffs, vals.cpu().numpy(), voffs)


def _split(e: Entries, parts: int):
    cuts = [e.n * i // parts for i in range(parts + 1)]
    for a, b in zip(cuts, cuts[1:]):
        if b > a:
            k0, v0 = e.koffs[a], e.voffs[a]
            yield Entries(e.keys[int(k0):int(e.koffs[b])], e.koffs[a:b + 1] - k0,
                          e.vals[int(v0):int(e.voffs[b])], e.voffs[a:b + 1] - v0)


def _options(c) -> TableOptions:
    return TableOptions(block_size=c["block"], restart_interval=c["restart"],
                        bits_per_key=c["bits"], max_file_size=c.get("max_file", 2 * MiB))


def _tables(g, c):
    """The job's files with their table bytes, the last sequence number."""
    opts, eng = _options(c), _engine()
    files = []

    def add(level, entries):
        data = eng.build_table(entries, opts)
        files.append(FileMeta(level, len(files) + 1, entries.key(0), entries.key(entries.n - 1),
                              len(data), None, data))

    n_low, n_up = c["lower"] * c["entries"], c["entries"]
    low = _distinct(g, n_low, c["klen"])
    runs = []  # upper runs: one per level-0 table, one in all below
    for _ in range(c["upper"] if c["level"] == 0 else 1):
        n = n_up if c["level"] == 0 else n_up * c["upper"]
        old = low[_perm(g, len(low))[:int(n * c["rewrite"])]]
        runs.append(torch.unique(torch.cat([old, _distinct(g, n - len(old), c["klen"])])))
    total = len(low) + sum(len(r) for r in runs)
    if c["level"] == 0:
        seqs = torch.cat([1 + sum(len(x) for x in [low] + runs[:i]) + _perm(g, len(r))
                          for i, r in enumerate([low] + runs) ])
        seqs[:len(low)] = 1 + _perm(g, len(low))
        at = len(low)
        for r in runs:
            seqs[at:at + len(r)] = at + 1 + _perm(g, len(r))
            at += len(r)
    else:
        # any order, but the upper version of a shared key is the newer one
        seqs = 1 + _perm(g, total)
        if len(low):
            up = runs[0]
            pos = torch.searchsorted(low, up).clamp(max=len(low) - 1)
            both = torch.nonzero(low[pos] == up).flatten()
            a, b = len(low) + both, pos[both]
            hi, lo = torch.maximum(seqs[a], seqs[b]), torch.minimum(seqs[a], seqs[b])
            seqs[a], seqs[b] = hi, lo
    if len(low):
        for e in _split(_entries(g, low, seqs[:len(low)], c), c["lower"]):
            add(c["level"] + 1, e)
    at = len(low)
    for r in runs:
        e = _entries(g, r, seqs[at:at + len(r)], c)
        at += len(r)
        for part in _split(e, 1 if c["level"] == 0 else c["upper"]):
            add(c["level"], part)
    return files, total


def _grandparents(files, c):
    """Files two levels down over the lower half of the key range (metadata only)."""
    k = c["grandparents"]
    if not k:
        return []
    keys = sorted({x[:-8] for f in files for x in (f.smallest, f.largest)})
    lo, hi = keys[0], keys[len(keys) // 2]
    a, b = (int.from_bytes(x[:8].ljust(8, b"\0"), "big") for x in (lo, hi))
    out, tag = [], (1 << 8 | 1).to_bytes(8, "little")
    step = max(2, (b - a) // k)
    for i in range(k):
        s = a + i * step
        out.append(FileMeta(c["level"] + 2, 100000 + i, s.to_bytes(8, "big") + tag,
                            (s + step // 2).to_bytes(8, "big") + tag, 2 * MiB))
    return out


def _on_device(tables):
    """The tables in one device buffer, back to back as a compaction leaves them."""
    total = sum(f.file_size for f in tables)
    buf = torch.empty(total + 64, dtype=torch.uint8, device="cuda")
    ptrs, at = [], 0
    for f in tables:
        buf[at:at + f.file_size] = torch.frombuffer(bytearray(f.data), dtype=torch.uint8).cuda()
        ptrs.append(buf.data_ptr() + at)
        at += f.file_size
        f.data = None
    return buf, ptrs


def _pinned(tables):
    for f in tables:
        t = torch.frombuffer(bytearray(f.data), dtype=torch.uint8).pin_memory()
        f.data = t.numpy()


def _prepare_compact(g, c):
    eng = _engine()
    if c["chained"]:
        return _prepare_chained(g, c)
    files, last = _tables(g, c)
    files += _grandparents(files, c)
    job = CompactionJob(c["level"], files, [last // 2] if c["snapshot"] else [], last, _options(c))
    tables = job.input_tables()
    if c["where"] == "host":
        _pinned(tables)
        return dict(job=eng.prepare(job, verify_checksums=c["verify"]), keep=[job])
    buf, ptrs = _on_device(tables)
    return dict(job=eng.prepare(job, ptrs, outputs_on_device=1, verify_checksums=c["verify"]),
                keep=[job, buf])


def _prepare_chained(g, c):
    """Level-1 inputs are an earlier compaction's outputs, kept decoded."""
    eng, opts = _engine(), _options(c)
    files, last = _tables(g, c)
    first = [f for f in files if f.level == 1]
    new = [f for f in files if f.level == 0]
    job1 = CompactionJob(1, first, [], last, opts)
    buf1, ptrs1 = _on_device(job1.input_tables())
    done = eng.run(eng.prepare(job1, ptrs1, outputs_on_device=1, keep_decoded=True))
    buf0, ptrs0 = _on_device(new)
    sizes = np.diff(done.file_offsets + [done.bytes_out])
    at = {f.number: (p, None) for f, p in zip(new, ptrs0)}
    for i, f in enumerate(done.files):
        new.append(FileMeta(1, 1000 + i, f.smallest, f.largest, int(sizes[i])))
        at[1000 + i] = (done.device_ptr + done.file_offsets[i], f.decoded)
    job = CompactionJob(0, new, [], last, opts)
    ptrs, decoded = zip(*[at[f.number] for f in job.input_tables()])
    prep = eng.prepare(job, list(ptrs), outputs_on_device=2, verify_checksums=c["verify"],
                       keep_decoded=True, decoded=list(decoded))
    return dict(job=prep, keep=[job, buf0, done])


def _batch_jobs(case):
    """The batch's job shapes: sizes log-uniform, 2-12 tables each."""
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["jobs"]):
        size = _log_int(r, case["lo_kib"], case["hi_kib"]) * KiB
        n = r.randint(2, 12)
        upper = r.randint(1, min(4, n - 1))
        out.append(_compact(upper=upper, lower=n - upper, vlen=case["vlen"],
                            entries=max(8, size // n // (case["vlen"] + 24))))
    return out


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind = case["kind"]
    if kind == "compact":
        state = dict(jobs=[_prepare_compact(g, case)])
    elif kind == "batch":
        state = dict(jobs=[_prepare_compact(g, c) for c in _batch_jobs(case)])
    elif kind == "flush":
        ids = _distinct(g, case["entries"], case["klen"])
        state = dict(entries=_entries(g, ids, 1 + _perm(g, len(ids)), case), opts=_options(case))
    else:
        n = case["size"] + case["offset"]
        buf = torch.randint(-(1 << 62), 1 << 62, (n // 8 + 1,), generator=g, device="cuda")
        state = dict(buf=buf, ptr=buf.data_ptr() + case["offset"], n=case["size"])
    torch.cuda.synchronize()  # the engine works on its own streams
    return dict(state, kind=kind)


# Where an output is cut, per case: its size depends on the seed a little, but what
# `run` returns has one shape per case.  The first `head` bytes are returned in place;
# the rest, up to `tail` bytes, in a zero-padded buffer beside them.
_cuts = {}


def _spread(c):
    """Six standard deviations of an output's relative size, generously."""
    n = c["entries"] * (c["upper"] + c["lower"] if "upper" in c else 1)
    cv = 0.05 + math.sqrt(c["tomb"]) + {"fixed": 0, "lognormal": 1.31, "loguniform": 0.8}[c["vdist"]]
    if c.get("snapshot"):
        cv += 0.5 * math.sqrt(c["rewrite"])
    return min(0.9, 0.001 + 6 * cv / math.sqrt(n))


def _cut_of(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _cuts:
        state = _inputs(case, 20011)
        shapes = _batch_jobs(case) if case["kind"] == "batch" else [case]
        sizes = [(r.bytes_out, len(r.files)) for r in _call(state)]
        cuts = []
        for c, (size, files) in zip(shapes, sizes):
            slack = int(size * _spread(c)) + 300 * files + 4096
            cuts.append((max(0, size - slack), 2 * slack))
        _cuts[key] = (cuts, int(1.1 * sum(f for _, f in sizes)) + 4 * len(sizes) + 4)
    return _cuts[key]


def prepare(case, seed):
    if case["kind"] == "crc":
        return _inputs(case, seed)
    cuts, files = _cut_of(case)
    state = _inputs(case, seed)
    on_device = state["kind"] == "batch" or case.get("where") == "device" and not case["chained"]
    room = sum(t for _, t in cuts)
    state["tail"] = (torch.zeros(room, dtype=torch.uint8, device="cuda") if on_device
                     else np.zeros(room, np.uint8))
    torch.cuda.synchronize()
    return dict(state, cuts=cuts, files=files)


# --------------------------------------------------------------------------
# one pass

class _View:
    """Output bytes of a result, without a copy; keeps the result alive."""

    def __init__(self, res):
        self.res = res
        if res.device_ptr and not len(res.files[0].data):
            self.__cuda_array_interface__ = dict(shape=(res.bytes_out,), typestr="|u1", version=2,
                                                 data=(res.device_ptr, False))
        else:
            first = np.frombuffer(res.files[0].data, np.uint8)
            self.__array_interface__ = dict(shape=(res.bytes_out,), typestr="|u1", version=3,
                                            data=(first.ctypes.data, False))


def _bytes(res):
    if isinstance(res, _Table):
        return np.frombuffer(res.data, np.uint8)
    if res.bytes_out == 0:
        return np.zeros(0, np.uint8)
    v = _View(res)
    return torch.as_tensor(v, device="cuda") if hasattr(v, "__cuda_array_interface__") else np.asarray(v)


class _Table:
    """A flushed table, as a result of one file."""

    def __init__(self, data):
        self.data, self.bytes_out, self.files = data, len(data), (None,)


def _call(state):
    eng = _engine()
    if state["kind"] == "flush":
        return [_Table(eng.build_table(state["entries"], state["opts"]))]
    if state["kind"] == "compact":
        return [eng.run(state["jobs"][0]["job"])]
    return eng.run_batch([j["job"] for j in state["jobs"]])


def _file_table(results, cap):
    """Every output file's offset and entry count, and its boundary keys."""
    nums = np.zeros(2 * cap, np.int64)
    got = [x for r in results for f, o in zip(r.files, r.file_offsets) for x in (o, f.entries)]
    nums[:len(got)] = got
    keys = b"".join(k for r in results for f in r.files for k in (f.smallest, f.largest))
    text = np.zeros(2 * 72 * cap, np.uint8)
    text[:len(keys)] = np.frombuffer(keys, np.uint8)
    return dict(files=nums, keys=text)


def run(state):
    if state["kind"] == "crc":
        return _engine().crc32c(device_ptr=state["ptr"], n=state["n"])
    results = _call(state)
    heads, dst, src, at = [], [], [], 0
    for res, (head, room) in zip(results, state["cuts"]):
        data = _bytes(res)
        assert head <= len(data) <= head + room, (head, len(data), room)
        heads.append(data[:head])
        dst.append(state["tail"][at:at + len(data) - head])
        src.append(data[head:])
        at += room
    if isinstance(state["tail"], np.ndarray):
        dst[0][:] = src[0]
    else:
        torch._foreach_copy_(dst, src)
    out = dict(data=heads, tail=state["tail"],
               sizes=np.array([r.bytes_out for r in results], np.int64))
    if state["kind"] != "flush":
        out.update(_file_table(results, state["files"]))
    return out


# --------------------------------------------------------------------------
# what a pass cannot do without

def _mean_value(c):
    if c["vdist"] == "lognormal":
        return c["vlen"] * math.exp(0.5)
    if c["vdist"] == "loguniform":
        return c["vlen"] * (4 - 1 / 4) / (2 * math.log(4))
    return c["vlen"]


def _entry_bytes(c):
    """A table's bytes per entry: the key without its shared prefix, tag, value, header."""
    shared = {16: 11, 8: 2, 24: 2, 0: 6}[c["klen"]] * (1 - 1 / c["restart"])
    return (c["klen"] or 36) - shared + 11 + _mean_value(c) * (1 - c["tomb"])


def _compact_bytes(c):
    tables = (c["upper"] + c["lower"]) * c["entries"]
    dropped = c["upper"] * c["entries"] * (c["rewrite"] if c["lower"] else 0)
    if c["snapshot"]:
        dropped /= 2
    return (2 * tables - dropped) * _entry_bytes(c)


def work(case):
    kind = case["kind"]
    if kind == "compact":
        b = _compact_bytes(case)
    elif kind == "batch":
        b = sum(_compact_bytes(c) for c in _batch_jobs(case))
    elif kind == "flush":
        raw = (case["klen"] or 36) + 8 + 16 + _mean_value(case) * (1 - case["tomb"])
        b = case["entries"] * (raw + _entry_bytes(case))
    else:
        b = case["size"]
    return {"bytes": float(b), "flops": 0.0}
