"""The span copy where its ways change: short and long spans side by side, calls of few and of many spans, parts of one
span, and spans of no bytes among them."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from cubam_b200 import _lib  # noqa: E402
from cubam_b200.bgzf import stream_ptr  # noqa: E402

MANY = 2 * 148 * 64  # spans from which a warp takes eight


@pytest.mark.parametrize("co_aligned", [True, False])
@pytest.mark.parametrize("n", [1, 3, 300, MANY // 4, MANY - 1, MANY, MANY + 5])
def test_copy_spans_of_every_length(n, co_aligned):
    rng = np.random.default_rng(n)
    longest = 2_000_003 if n <= 3 else 3000
    sizes = np.array([*range(0, 40), 255, 256, 257, 258, 511, 512, 513, 527, 528, 1000, longest, -1, -1000])
    size = sizes[rng.integers(0, len(sizes), n)]
    size[rng.integers(0, n)] = longest
    some = np.maximum(size, 0)
    off = rng.integers(0, 4_000_000 - some + 1)
    off[size <= 0] = 4_000_000
    dst = np.cumsum(some + 40) - some  # 40 bytes between
    if co_aligned:
        dst += (off - dst) % 16
    src = torch.randint(0, 256, (4_000_000,), dtype=torch.uint8, device="cuda")
    out = torch.full((int(dst[-1] + some[-1]) + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    o, d, s = (torch.from_numpy(x.astype(np.int64)).cuda() for x in (off, dst, size))
    assert _lib.lib.cb_copy_spans(src.data_ptr(), out.data_ptr(), o.data_ptr(), d.data_ptr(), s.data_ptr(), n,
                                  stream_ptr()) == 0
    data, got = src.cpu().numpy(), out.cpu().numpy()
    want = np.full(len(got), 0xA5, np.uint8)
    for a, b, k in zip(off, dst, some, strict=True):
        want[b : b + k] = data[a : a + k]
    assert np.array_equal(got, want)
