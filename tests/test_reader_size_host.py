"""The reader's chunks where a file changes as it is opened (without CUDA: host chunks)."""

import os

import pytest

torch = pytest.importorskip("torch")
if torch.cuda.is_available():
    pytest.skip("the host form of the reader", allow_module_level=True)


@pytest.mark.parametrize("before", [None, b"", b"0123456789"], ids=["missing", "empty", "short"])
def test_chunks_are_of_the_opened_file(tmp_path, monkeypatch, before):
    from cubam_b200.bgzf import _ChunkReader

    p = tmp_path / "growing"
    if before is not None:
        p.write_bytes(before)
    data = bytes(range(256)) * 40
    real = os.open

    def grow(path, *args, **kw):
        if os.fspath(path) == str(p):
            p.write_bytes(data)
        return real(path, *args, **kw)

    monkeypatch.setattr(os, "open", grow)
    chunks = [(c.numpy().tobytes(), eof) for c, eof in _ChunkReader(p, 4096)]
    assert [(len(c), eof) for c, eof in chunks] == [(4096, False), (4096, False), (2048, True)]
    assert b"".join(c for c, _ in chunks) == data


def test_what_is_written_later_is_not_read(tmp_path):
    from cubam_b200.bgzf import _ChunkReader

    p = tmp_path / "appended"
    p.write_bytes(b"x" * 5000)
    r = _ChunkReader(p, 4096)
    with p.open("ab") as f:
        f.write(b"y" * 5000)
    assert b"".join(c.numpy().tobytes() for c, _ in r) == b"x" * 5000


def test_files_are_closed(tmp_path):
    from cubam_b200.bgzf import _ChunkReader

    p = tmp_path / "f"
    p.write_bytes(b"x" * 5000)
    fds = set(os.listdir("/proc/self/fd"))
    for _ in range(3):
        r = _ChunkReader(p, 4096)
        assert len(list(r)) == 2
        r._thread.join()
    assert set(os.listdir("/proc/self/fd")) == fds
