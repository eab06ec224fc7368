"""The two-range form of the split inflater from several threads and streams, also while one of them captures."""

import threading
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from cubam_b200 import _lib, bgzf as G  # noqa: E402

RANGES = 20 * 148 + 40  # jobs that go in two ranges


class _Members:
    """``n`` members of a few bytes each and all that a call of them needs."""

    def __init__(self, n, seed):
        rng = np.random.default_rng(seed)
        blob, rows, want, off = bytearray(), [], [], 0
        for _ in range(64):
            data = rng.choice(np.frombuffer(b"ACGT\n", np.uint8), int(rng.integers(1, 90))).tobytes()
            raw = zlib.compress(data, 6)[2:-4]
            blob += bytes(18)
            rows.append([len(blob), 0, len(raw) | (len(data) << 32), zlib.crc32(data)])
            blob += raw + bytes(8)
            want.append(np.frombuffer(data, np.uint8))
        pick = rng.integers(0, 64, n)
        self.buf = torch.frombuffer(blob, dtype=torch.uint8).cuda()
        table = np.array(rows, dtype=np.int64)[pick]
        size = table[:, 2] >> 32
        table[:, 0] += self.buf.data_ptr()
        table[:, 1] = np.cumsum(size) - size
        self.n, self.total = n, int(size.sum())
        self.want = np.concatenate([want[k] for k in pick])
        self.table = torch.from_numpy(table).cuda()
        self.out = torch.zeros(self.total, dtype=torch.uint8, device="cuda")
        self.summ = torch.zeros(G.ctypes_sizeof(_lib.InflateSummary), dtype=torch.uint8, device="cuda")
        self.ws = torch.empty(G.inflate_workspace_bytes(n, self.total, 3), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def launch(self):
        G.launch_inflate(self.table.data_ptr(), self.n, self.out.data_ptr(), self.total, True, self.summ.data_ptr(), self.ws, 3)

    def check(self):
        assert G.read_struct(self.summ, _lib.InflateSummary).status == _lib.OK
        assert np.array_equal(self.out.cpu().numpy(), self.want)


@pytest.mark.parametrize("jobs", [65_536, 400])
def test_one_thread_captures_while_another_decodes(jobs):
    """A graph of two ranges (at any size with the pipeline always on) is recorded on one thread; a call that goes in two
    ranges runs on another meanwhile; both give their members' bytes, and so does a call on the first stream after."""
    captured, eager = _Members(jobs, 1), _Members(RANGES, 2)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        captured.launch()
    a.synchronize()
    captured.out.zero_()
    torch.cuda.synchronize()
    open_, done, failure = threading.Event(), threading.Event(), []

    def other():
        try:
            assert open_.wait(60)
            with torch.cuda.stream(b):
                eager.launch()
        except BaseException as e:  # noqa: BLE001
            failure.append(e)
        finally:
            done.set()

    t = threading.Thread(target=other)
    t.start()
    g = torch.cuda.CUDAGraph()
    if jobs < 65_536:
        _lib.lib.cb_set_param(_lib.PARAM_DECODE_PIPELINE, 2)
    try:
        with torch.cuda.graph(g, stream=a, capture_error_mode="thread_local"):
            captured.launch()
            open_.set()
            assert done.wait(60)
    finally:
        _lib.lib.cb_set_param(_lib.PARAM_DECODE_PIPELINE, -1)
        open_.set()
        t.join()
    assert not failure, failure
    g.replay()
    torch.cuda.synchronize()
    captured.check()
    eager.check()
    captured.out.zero_()
    with torch.cuda.stream(a):
        captured.launch()
    torch.cuda.synchronize()
    captured.check()


def test_calls_on_more_streams_than_pairs():
    """Every stream's calls give their bytes, in order, whatever streams the others use."""
    streams = [torch.cuda.Stream() for _ in range(11)]
    members = [_Members(RANGES + 7 * k, 10 + k) for k in range(11)]
    for _ in range(3):
        for s, m in zip(streams, members, strict=True):
            with torch.cuda.stream(s):
                m.out.zero_()
                m.launch()
    torch.cuda.synchronize()
    for m in members:
        m.check()


def test_threads_share_the_pairs():
    members = [_Members(RANGES, 30 + k) for k in range(4)]
    failure = []

    def run(m):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    m.launch()
                torch.cuda.current_stream().synchronize()
        except BaseException as e:  # noqa: BLE001
            failure.append(e)

    threads = [threading.Thread(target=run, args=(m,)) for m in members]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failure, failure
    for m in members:
        m.check()
