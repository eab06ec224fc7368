"""The decoders that read a span of bytes by words (copies, hashes, packed bases), where spans begin and end at
every alignment, at an allocation's ends, and around the longest that four lanes copy."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from cubam_b200 import _lib  # noqa: E402
from cubam_b200.bgzf import stream_ptr  # noqa: E402
from oracle import bam_oracle as O  # noqa: E402


def _spans(n_bytes):
    rng = np.random.default_rng(3)
    sizes = [*range(0, 14), 15, 16, 17, 31, 32, 33, 63, 65, 511, 512, 513, 2001]
    off = [(int(rng.integers(0, (n_bytes - n) // 4)) * 4 + a) % (n_bytes - n + 1) for n in sizes for a in range(4)]
    size = [n for n in sizes for _ in range(4)]
    for n in (1, 2, 3, 5, 6):  # at the ends of the buffer
        off += [0, n_bytes - n]
        size += [n, n]
    return np.array(off, np.int64), np.array(size, np.int64)


def _fnv(b):
    x = 1469598103934665603
    for c in b:
        x = ((x ^ c) * 1099511628211) % (1 << 64)
    return x


@pytest.mark.parametrize("gap", [0, 1, 2, 3])
def test_copy_spans(gap):
    data = np.random.default_rng(1).integers(0, 256, 4099, dtype=np.uint8)
    off, size = _spans(len(data))
    dst = gap + np.cumsum(size + gap) - size - gap
    total = int(dst[-1] + size[-1])
    src = torch.from_numpy(data).cuda()
    out = torch.full((total,), 0xA5, dtype=torch.uint8, device="cuda")
    o, d, s = (torch.from_numpy(x).cuda() for x in (off, dst, size))
    assert _lib.lib.cb_copy_spans(src.data_ptr(), out.data_ptr(), o.data_ptr(), d.data_ptr(), s.data_ptr(), len(off),
                                  stream_ptr()) == 0
    want = np.full(total, 0xA5, np.uint8)
    for a, b, n in zip(off, dst, size, strict=True):
        want[b : b + n] = data[a : a + n]
    assert out.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("kind", ["bytes", "bases"])
def test_hash_and_pack_of_spans(kind):
    rng = np.random.default_rng(2)
    data = rng.integers(0, 256, 4099, dtype=np.uint8)
    if kind == "bases":
        data = rng.choice(np.frombuffer(b"ACGTACGTACGTACGTACGTACGTACGT-1-0N", np.uint8), 4099)
    off, size = _spans(len(data))
    src, o, n = torch.from_numpy(data.copy()).cuda(), torch.from_numpy(off).cuda(), torch.from_numpy(size.astype(np.int32)).cuda()
    h = torch.empty(len(off), dtype=torch.int64, device="cuda")
    code, ok = torch.empty_like(h), torch.empty(len(off), dtype=torch.uint8, device="cuda")
    assert _lib.lib.cb_hash_spans(src.data_ptr(), o.data_ptr(), n.data_ptr(), len(off), h.data_ptr(), stream_ptr()) == 0
    assert _lib.lib.cb_pack_acgt(src.data_ptr(), o.data_ptr(), n.data_ptr(), len(off), code.data_ptr(), ok.data_ptr(),
                                 stream_ptr()) == 0
    raw = data.tobytes()
    assert h.cpu().numpy().view(np.uint64).tolist() == [_fnv(raw[a : a + k]) for a, k in zip(off, size, strict=True)]
    want, fits = O.pack_acgt(raw, off, size)
    assert code.cpu().numpy().view(np.uint64).tolist() == [int(x) for x in want]
    assert [bool(x) for x in ok.cpu().tolist()] == [bool(x) for x in fits]
