"""The split inflater (decode of 32 segments at once, copy by rounds, CRC32 by rows) against zlib where its
tiles, windows and slots have edges."""

import random
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from cubam_b200 import _lib, bgzf as G  # noqa: E402

BLOCK = 0xFF00


def _raw(data, level=6, strategy=zlib.Z_DEFAULT_STRATEGY, flush_every=0, mem=8):
    z = zlib.compressobj(level, zlib.DEFLATED, -15, mem, strategy)
    if not flush_every:
        return z.compress(data) + z.flush()
    parts = [z.compress(data[i : i + flush_every]) + z.flush(zlib.Z_FULL_FLUSH) for i in range(0, len(data), flush_every)]
    return b"".join(parts) + z.flush()


def _edges():
    """Sizes at the edges of words, lines (128), CRC rows (4096) and members, as text, noise and runs."""
    rng = random.Random(5)
    out = []
    for n in (1, 2, 3, 4, 5, 31, 32, 127, 128, 129, 255, 256, 257, 4093, 4095, 4096, 4097, 4100, 8191, 8193, BLOCK):
        text = bytes(rng.choices(b"ACGT\n0123", k=n))
        noise = rng.randbytes(n)
        for p, kw in ((text, {}), (noise, {}), (b"x" * n, {}), (text, {"strategy": zlib.Z_FIXED}),
                      (noise, {"strategy": zlib.Z_HUFFMAN_ONLY}), (text, {"level": 0})):
            out.append((p, kw))
    return out


def _distances():
    """Matches from just inside to just outside each window of the copy, and that overlap themselves."""
    rng = random.Random(6)
    out = []
    for d in (1, 2, 3, 7, 8, 31, 127, 128, 129, 4095 - 1280, 4096, 8192 - 1280, 8192, 16384, 32767, 32768):
        base = rng.randbytes(d)
        out.append((base * (BLOCK // d) + base[: BLOCK % d], {}))
        mixed = bytearray(base)
        while len(mixed) < BLOCK - 300:  # short matches among literals
            k = rng.randint(3, 40)
            mixed += bytes(mixed[-d + i % d] for i in range(k)) + rng.randbytes(rng.randint(0, 3))
        out.append((bytes(mixed), {"level": 9}))
    return out


def _blocks():
    """Many blocks per member, down to ones whose runs do not fit the member's slot, and skewed codes."""
    rng = random.Random(7)
    text = bytes(rng.choices(b"ACGTN\tchr12345", k=BLOCK))
    out = [(text[:30000], {"flush_every": k}) for k in (7, 40, 300, 2000, 9000)]
    skew = bytes(rng.choices(range(64), weights=[1.0 / (1 << min(i, 20)) for i in range(64)], k=BLOCK // 2))
    out.append((skew + rng.randbytes(BLOCK // 2 - 200), {"strategy": zlib.Z_HUFFMAN_ONLY}))
    out.append((skew * 2, {"strategy": zlib.Z_HUFFMAN_ONLY}))
    out.append((text, {"mem": 1}))
    fib = [1, 1]
    while len(fib) < 24:
        fib.append(fib[-1] + fib[-2])
    deep = [b for i, f in enumerate(fib) for b in [i * 11 % 256] * min(f, 9000)][: BLOCK]  # codes of all lengths
    rng.shuffle(deep)
    out.append((bytes(deep), {"strategy": zlib.Z_HUFFMAN_ONLY}))
    return out


def _table(cases, out_shift=0, gap=0):
    """The members' bytes on the GPU and their job table (``gap`` unused bytes after each member's output)."""
    blob, rows, off = bytearray(), [], out_shift
    for data, kw in cases:
        raw = _raw(data, **kw)
        blob += bytes(18)
        rows.append([len(blob), off, len(raw) | (len(data) << 32), zlib.crc32(data)])
        blob += raw + zlib.crc32(data).to_bytes(4, "little") + len(data).to_bytes(4, "little")
        off += len(data) + gap
    buf = torch.frombuffer(blob, dtype=torch.uint8).cuda()
    table = np.array(rows, dtype=np.int64)
    table[:, 0] += buf.data_ptr()
    return buf, torch.from_numpy(table).cuda(), off


def _run(table, total, workspace_bytes, form, check_crc=True):
    out = torch.full((total + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    summ = torch.zeros(G.ctypes_sizeof(_lib.InflateSummary), dtype=torch.uint8, device="cuda")
    codes = torch.full((len(table),), 99, dtype=torch.int32, device="cuda")
    ws = torch.empty(workspace_bytes, dtype=torch.uint8, device="cuda")
    G.launch_inflate(table.data_ptr(), len(table), out.data_ptr(), total, check_crc, summ.data_ptr(), ws, form,
                     codes.data_ptr())
    return out.cpu().numpy(), codes.cpu().numpy(), G.read_struct(summ, _lib.InflateSummary)


@pytest.mark.parametrize("window", [6, 12, 24])
@pytest.mark.parametrize("make", [_edges, _distances, _blocks], ids=["edges", "distances", "blocks"])
def test_split_matches_zlib(make, window):
    cases = make()
    want = b"".join(d for d, _ in cases)
    assert _lib.lib.cb_set_param(_lib.PARAM_COPY_WARPS, window) == 0
    try:
        for shift in (0, 5):
            buf, table, total = _table(cases, shift)
            out, codes, summ = _run(table, total, G.inflate_workspace_bytes(len(cases), total, 3), 3)
            assert summ.status == 0 and summ.n_bad == 0 and summ.first_bad == -1 and not codes.any()
            assert out[shift:total].tobytes() == want
            assert (out[:shift] == 0xA5).all() and (out[total:] == 0xA5).all()
    finally:
        _lib.lib.cb_set_param(_lib.PARAM_COPY_WARPS, -1)


@pytest.mark.parametrize("jobs,window", [(400, -1), (600, -1), (1100, -1), (2100, 6), (2100, 12), (2100, 24), (3100, 12)])
@pytest.mark.parametrize("make", [_edges, _distances, _blocks], ids=["edges", "distances", "blocks"])
def test_split_matches_zlib_at_every_width(make, jobs, window):
    """The same members many times over: members take 4, 2 and 1 warps as the calls hold more
    of them, and then go in two ranges."""
    cases = make()
    times = -(-jobs // len(cases))
    buf, table, total = _table(cases, 3)
    rows = table.cpu().numpy()
    total -= 3
    many = np.concatenate([rows + np.array([0, k * total, 0, 0]) for k in range(times)])
    _lib.lib.cb_set_param(_lib.PARAM_COPY_WARPS, window)
    try:
        size = G.inflate_workspace_bytes(len(many), times * total, 3)
        out, codes, summ = _run(torch.from_numpy(many).cuda(), 3 + times * total, size, 3)
    finally:
        _lib.lib.cb_set_param(_lib.PARAM_COPY_WARPS, -1)
    assert summ.status == 0 and summ.n_bad == 0 and not codes.any()
    want = np.frombuffer(b"".join(d for d, _ in cases), dtype=np.uint8)
    assert (out[3 : 3 + times * total].reshape(times, total) == want).all()
    assert (out[:3] == 0xA5).all() and (out[3 + times * total :] == 0xA5).all()


def test_split_reports_crc_and_size():
    """A wrong CRC32 (also unchecked), and an ISIZE one too small or too large, in members of every size."""
    cases = [(d, kw) for d, kw in _edges() if len(d) > 1][::5]
    buf, table, total = _table(cases, gap=1)  # room for the ISIZE that is one too large
    rows = table.cpu().numpy().copy()
    rows[0::4, 3] ^= 1
    rows[1::4, 2] -= 1 << 32
    rows[2::4, 2] += 1 << 32
    bad = torch.from_numpy(rows).cuda()
    size = G.inflate_workspace_bytes(len(cases), total + len(cases), 3)
    kinds = np.arange(len(cases)) % 4
    want = np.array([_lib.CRC, _lib.INFLATE, _lib.INFLATE, _lib.OK])[kinds]
    out, codes, summ = _run(bad, total, size, 3)
    assert codes.tolist() == want.tolist()
    assert summ.n_bad == int((want != 0).sum()) and summ.first_bad == 0 and summ.status == _lib.CRC
    _, codes, _ = _run(bad, total, size, 3, check_crc=False)
    assert codes.tolist() == np.where(want == _lib.CRC, _lib.OK, want).tolist()


@pytest.mark.parametrize("room", ["small", "head", "half", "full", "odd"])
def test_any_workspace_for_few_jobs(room):
    """A call of few jobs that leaves the form to the library takes every workspace from 256 bytes up."""
    cases = _edges()
    buf, table, total = _table(cases)
    full = int(_lib.lib.cb_inflate_split_workspace_bytes(len(cases), total))
    size = {"small": 256, "head": 256 + 16 * len(cases) + 600, "half": full - total, "full": full, "odd": full + 9}[room]
    out, codes, summ = _run(table, total, size, 0)
    assert summ.status == 0 and not codes.any()
    assert out[:total].tobytes() == b"".join(d for d, _ in cases)


def test_split_workspace_too_small_is_an_error():
    """Form 3 asked for by name: the jobs whose slots the workspace does not hold fail, the others do not."""
    cases = [c for c in _edges() if len(c[0]) >= 4093]
    buf, table, total = _table(cases)
    full = int(_lib.lib.cb_inflate_split_workspace_bytes(len(cases), total))
    out, codes, summ = _run(table, total, full - total, 3)
    assert set(codes.tolist()) == {_lib.OK, _lib.CAPACITY} and codes[0] == 0 and codes[-1] == _lib.CAPACITY
    assert summ.status == _lib.CAPACITY
    assert out[: len(cases[0][0])].tobytes() == cases[0][0]


@pytest.mark.parametrize("jobs", [30, 400, 700, 1300, 3100])
def test_stored_members(jobs):
    """Members of one or several stored blocks, alone and before or after coded ones, at every width."""
    rng = random.Random(8)
    noise = rng.randbytes(BLOCK)
    text = bytes(rng.choices(b"ACGT\n0123", k=9000))
    cases = [(noise, {"level": 0}), (noise, {}), (noise[:40_000], {"mem": 1}), (noise[:20_000], {"level": 0, "flush_every": 700}),
             (noise[:20_000] + text, {}), (text + noise[:20_000], {}), (noise[:1], {"level": 0}), (text, {})]
    times = -(-jobs // len(cases))
    buf, table, total = _table(cases, 3)
    rows = table.cpu().numpy()
    total -= 3
    many = np.concatenate([rows + np.array([0, k * total, 0, 0]) for k in range(times)])
    size = G.inflate_workspace_bytes(len(many), times * total, 3)
    out, codes, summ = _run(torch.from_numpy(many).cuda(), 3 + times * total, size, 3)
    assert summ.status == 0 and not codes.any()
    want = np.frombuffer(b"".join(d for d, _ in cases), dtype=np.uint8)
    assert (out[3 : 3 + times * total].reshape(times, total) == want).all()
    many[:, 3] ^= np.arange(len(many)) % 3 == 1  # a wrong CRC32
    _, codes, summ = _run(torch.from_numpy(many).cuda(), 3 + times * total, size, 3)
    assert (codes == np.where(np.arange(len(many)) % 3 == 1, _lib.CRC, _lib.OK)).all()


@pytest.mark.parametrize("jobs", [40, 400, 800, 3100])
def test_jobs_may_share_their_output(jobs):
    """Every member twice in a call, with one place for both; and places that are read while they are written again."""
    rng = random.Random(9)
    cases = [(bytes(rng.choices(b"ACGT\n0123", k=rng.choice([900, 9000, BLOCK]))), {"level": rng.choice([1, 6])}) for _ in range(20)]
    buf, table, total = _table(cases)
    rows = table.cpu().numpy()
    half = jobs // 2
    many = np.concatenate([rows + np.array([0, k * total, 0, 0]) for k in range(-(-half // len(cases)))])[:half]
    both = torch.from_numpy(np.concatenate([many, many[::-1]])).cuda()
    n = int(many[-1, 1] + (many[-1, 2] >> 32))
    want = np.frombuffer(b"".join(d for d, _ in cases) * (len(many) // len(cases) + 1), dtype=np.uint8)[:n]
    out = torch.full((n,), 0xA5, dtype=torch.uint8, device="cuda")
    seen = torch.empty_like(out)
    summ = torch.zeros(G.ctypes_sizeof(_lib.InflateSummary), dtype=torch.uint8, device="cuda")
    ws = torch.empty(G.inflate_workspace_bytes(len(both), 2 * n, 3), dtype=torch.uint8, device="cuda")
    reader = torch.cuda.Stream()
    for k in range(3):
        G.launch_inflate(both.data_ptr(), len(both), out.data_ptr(), 2 * n, True, summ.data_ptr(), ws, 3)
        assert G.read_struct(summ, _lib.InflateSummary).status == 0
        assert np.array_equal(out.cpu().numpy(), want)
        G.launch_inflate(both.data_ptr(), len(both), out.data_ptr(), 2 * n, True, summ.data_ptr(), ws, 3)
        with torch.cuda.stream(reader):
            seen.copy_(out)
        torch.cuda.synchronize()
        assert np.array_equal(seen.cpu().numpy(), want)


def _damaged():
    """Members of up to 65 KB with bits flipped in their headers, code lengths and symbols, cut short, or of another size or
    CRC32 than said: (raw stream, size said, CRC32 said)."""
    rng = random.Random(12)
    text = b"".join(bytes(rng.choices(b"ACGTN\tchr12345:,;\n", k=40)) * rng.choice([1, 1, 2]) for _ in range(1200))[:BLOCK]
    skew = bytes(rng.choices(range(64), weights=[1.0 / (1 << min(i, 20)) for i in range(64)], k=BLOCK))
    bases = [(text, {}), (text, {"level": 1, "mem": 1}), (text, {"strategy": zlib.Z_FIXED}), (skew, {"strategy": zlib.Z_HUFFMAN_ONLY}),
             (rng.randbytes(BLOCK), {}), (text[:30_000], {"flush_every": 3000})]
    out = []
    for data, kw in bases:
        raw = _raw(data, **kw)
        for region in ((0, 4), (4, 90), (90, len(raw) // 2), (len(raw) // 2, len(raw)), (len(raw) - 6, len(raw))):
            for _ in range(3):
                bad = bytearray(raw)
                for _ in range(rng.randint(1, 3)):
                    bad[rng.randrange(*region)] ^= 1 << rng.randrange(8)
                out.append((bytes(bad), len(data), zlib.crc32(data)))
        out.append((raw[: len(raw) * 2 // 3], len(data), zlib.crc32(data)))
        out.append((raw[:40], len(data), zlib.crc32(data)))
        out.append((raw, len(data) - 1, zlib.crc32(data)))
        out.append((raw, len(data) // 2, zlib.crc32(data)))
        out.append((raw, len(data) + 1, zlib.crc32(data)))
        out.append((raw, len(data), zlib.crc32(data) ^ 1))
    return out, [(_raw(d, **kw), len(d), zlib.crc32(d)) for d, kw in bases], [d for d, _ in bases]


@pytest.mark.parametrize("jobs", [60, 400, 800, 1500, 3200])
def test_damaged_members_at_every_width(jobs):
    """Damaged members among good ones, at 8, 4, 2 and 1 warps per member and in two ranges: the codes of the one-kernel form,
    the good members' bytes, and nothing written between the members' outputs."""
    bad, good, data = _damaged()
    gap, rng = 5, np.random.default_rng(jobs)
    blob, at, rows, off = bytearray(), {}, [], 3
    kinds = np.where(rng.random(jobs) < 0.5, rng.integers(0, len(bad), jobs), -1 - rng.integers(0, len(good), jobs))
    for k in kinds.tolist():
        raw, size, crc = bad[k] if k >= 0 else good[-1 - k]
        if k not in at:
            blob += bytes(18)
            at[k] = len(blob)
            blob += raw + bytes(8)
        rows.append([at[k], off, len(raw) | (size << 32), crc])
        off += size + gap
    buf = torch.frombuffer(blob, dtype=torch.uint8).cuda()
    table = np.array(rows, dtype=np.int64)
    table[:, 0] += buf.data_ptr()
    table = torch.from_numpy(table).cuda()
    results = {}
    for form in (1, 3):
        out, codes, summ = _run(table, off, G.inflate_workspace_bytes(jobs, off, form), form)
        assert summ.n_bad == int((codes != 0).sum()) and summ.first_bad == int(np.flatnonzero(codes)[0])
        results[form] = codes, int(summ.status)
        between = np.ones(len(out), dtype=bool)
        for k, (_, o, w, _), code in zip(kinds.tolist(), rows, codes.tolist(), strict=True):
            between[o : o + (w >> 32)] = False
            if k < 0:
                assert code == 0 and out[o : o + (w >> 32)].tobytes() == data[-1 - k]
        assert (out[between] == 0xA5).all()
    assert (results[1][0] == results[3][0]).all() and results[1][1] == results[3][1]
    assert set(results[3][0].tolist()) == {_lib.OK, _lib.INFLATE, _lib.CRC}
