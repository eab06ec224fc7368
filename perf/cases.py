"""The work this package does for its users, as cases that can be timed.

A case names one call of the public API on one input: a BAM file decoded from GPU memory
(``decode_resident``, ``decode_many``, a captured ``BatchPlan``), read from the file system
(``read_bam``), the columns, tags and on-request decoders of its records (``RecordBatch``), or the
BGZF writer's compression (``bgzf._bgzf_compress``).  Inputs are seeded synthetic BAM files of the
three benchmark shapes (``cubam_b200.synth``: ``small`` single-end 90 bp reads with CB/UB tags,
``gex`` spliced 91 bp reads with five tags, ``atac`` 50 bp pairs).  Files of more than
``UNIT_RECORDS`` records repeat the BGZF members of a file of that size, so that making them stays
quick; every member is still inflated and every record decoded on its own.

- ``listed()``: the cases; ``draw(rng)``: another one of the same ranges.
- ``prepare(case, seed)``: the input and what a program keeps for it; ``run(state)``: one call.
- ``work(case)``: the bytes one call cannot do without.

All outputs are whole numbers and bytes.
"""

import math
import os
import shutil
import struct
import tempfile
import zlib
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import cubam_b200
from cubam_b200 import batch, bgzf, synth
from cubam_b200.bam import FIELDS, RecordBatch

UNIT_RECORDS = 250_000
RUN = 500  # records that keep their order: about two BGZF blocks
SHAPES = {"small": 0, "gex": 1, "atac": 2}
#: bytes of a record, inflated and in a file of zlib level 6
RECORD = {"small": (230.0, 135.2), "gex": (252.2, 101.0), "atac": (154.0, 55.9)}
TAGS = {"small": ("CB", "UB"), "gex": ("CB", "UB", "GN"), "atac": ("CB",)}
COLUMN_BYTES = 8 + 7 * 4 + 1 + 3 * 2  # a record's offset and its eleven columns
TAG_BYTES = 1 + 8 + 4 + 8


def listed():
    return [
        # one small file of a batch, or one region's worth of members: the call a server makes most
        {"name": "resident-gex-10k", "kind": "resident", "shape": "gex", "records": 10_000},
        # the whole of a small file (the package's own `small` workload)
        {"name": "resident-small-100k", "kind": "resident", "shape": "small", "records": 100_000},
        # a sample's worth of reads, both benchmark shapes
        {"name": "resident-gex-1m", "kind": "resident", "shape": "gex", "records": 1_000_000},
        {"name": "resident-atac-1m", "kind": "resident", "shape": "atac", "records": 1_000_003},
        # a whole run resident on the GPU: more members than the decoders hold in flight
        {"name": "resident-gex-18m", "kind": "resident", "shape": "gex", "records": 18_000_000},
        # files of very uneven sizes in one call, their members compressed at levels 1-9, some stored
        {"name": "many-uneven-6", "kind": "many", "files": 6, "low": 10_000, "high": 600_000},
        # a fixed batch decoded again and again as one CUDA graph
        {"name": "plan-gex-200k", "kind": "plan", "shape": "gex", "records": 200_000},
        # the reader on a path: a small file with the default chunk, a larger one in chunks
        {"name": "read-small-100k", "kind": "read", "shape": "small", "records": 100_000, "chunk": 0},
        {"name": "read-gex-2m-80mb", "kind": "read", "shape": "gex", "records": 2_000_000, "chunk": 80 << 20},
        # what an application asks of a batch of records: columns, tags, strings, hashes, blocks
        {"name": "records-gex-1m", "kind": "records", "shape": "gex", "records": 1_000_000},
        # the writer: one flush of it (1024 blocks) at its default level, and a large odd one
        {"name": "compress-gex-64mb", "kind": "compress", "shape": "gex", "bytes": 1024 * bgzf.BLOCK_DATA, "level": 2},
        {"name": "compress-gex-240mb", "kind": "compress", "shape": "gex", "bytes": 240_000_007, "level": 2},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["resident", "resident", "resident", "many", "plan", "read", "records", "compress"])
    shape = rng.choice(["small", "gex", "gex", "atac"])
    if kind == "resident":
        return {"kind": kind, "shape": shape, "records": _log_uniform(rng, 300, 12_000_000)}
    if kind == "many":
        return {"kind": kind, "files": rng.randint(2, 6), "low": _log_uniform(rng, 1_000, 20_000),
                "high": _log_uniform(rng, 50_000, 600_000)}
    if kind == "plan":
        return {"kind": kind, "shape": shape, "records": _log_uniform(rng, 1_000, 2_000_000)}
    if kind == "read":
        n = _log_uniform(rng, 1_000, 2_000_000)
        return {"kind": kind, "shape": shape, "records": n,
                "chunk": rng.choice([0, int(n * RECORD[shape][1] * rng.uniform(0.4, 1.2)) + 200_000])}
    if kind == "records":
        return {"kind": kind, "shape": shape, "records": _log_uniform(rng, 300, 2_000_000)}
    return {"kind": kind, "shape": shape, "bytes": _log_uniform(rng, 2_000, 200_000_000), "level": rng.choice([0, 1, 2, 2, 6])}


# ---------------------------------------------------------------- inputs

_base = {}


def _base_records(shape, n):
    """The header bytes and n records of a generated file: (header, its bytes, record bytes, record offsets)."""
    if (shape, n) not in _base:
        folder = tempfile.mkdtemp(prefix="cubam_cases_")
        try:
            path = os.path.join(folder, "base.bam")
            synth.write_bam(path, synth.Config("case", SHAPES[shape], n, 7, level=1,
                                               n_barcodes=10_000 if shape == "atac" else 1000))
            header = cubam_b200.BamHeader.read(path)
            raw = np.fromfile(path, dtype=np.uint8).tobytes()
        finally:
            shutil.rmtree(folder, ignore_errors=True)
        parts, at = [], 0
        while at < len(raw):
            size = int.from_bytes(raw[at + 16 : at + 18], "little") + 1
            parts.append(zlib.decompress(raw[at + 18 : at + size - 8], -15))
            at += size
        plain = b"".join(parts)
        records, offset, at = plain[header.size :], [], 0
        while at < len(records):
            offset.append(at)
            at += 4 + int.from_bytes(records[at : at + 4], "little")
        _base[shape, n] = header, plain[: header.size], records, offset
    return _base[shape, n]


def _shuffled(shape, n, seed):
    """About n records: runs of RUN records of the generated file in an order of the seed's own (so that
    inputs of two seeds differ while their sizes do not), repeated ``k`` times; (header, header bytes,
    record bytes, k)."""
    k = max(1, -(-n // UNIT_RECORDS))
    header, head, records, offset = _base_records(shape, max(n // k, 2))
    run = min(RUN, max(1, len(offset) // 8))
    starts = offset[::run] + [len(records)]
    order = np.random.RandomState(seed).permutation(len(starts) - 1)
    return header, head, b"".join(records[starts[i] : starts[i + 1]] for i in order), k


def _member(data, level):
    z = zlib.compressobj(level, zlib.DEFLATED, -15, 8)
    body = z.compress(data) + z.flush()
    return (bgzf.EOF_BLOCK[:16] + struct.pack("<H", len(body) + 25) + body + struct.pack("<II", zlib.crc32(data), len(data)))


def _bam(shape, n, seed, mixed=False):
    """A BAM file of about n records: its header and its bytes (uint8).  zlib level 6; with ``mixed``
    levels 1-9 at random per member and one member in fifty stored."""
    header, head, records, k = _shuffled(shape, n, seed)
    cuts = [records[a : a + bgzf.BLOCK_DATA] for a in range(0, len(records), bgzf.BLOCK_DATA)]
    rng = np.random.RandomState(seed)
    levels = [0 if mixed and rng.rand() < 0.02 else rng.randint(1, 10) if mixed else 6 for _ in cuts]
    with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
        body = b"".join(pool.map(_member, cuts, levels))
    return header, np.frombuffer(_member(head, 6) + body * k + bgzf.EOF_BLOCK, dtype=np.uint8)


def _resident(*args, **kw):
    header, raw = _bam(*args, **kw)
    return torch.from_numpy(raw.copy()).cuda(), header


class _File:
    """A file that goes away with the state that holds it."""

    def __init__(self, raw):
        self.folder = tempfile.mkdtemp(prefix="cubam_cases_")
        self.path = os.path.join(self.folder, "reads.bam")
        raw.tofile(self.path)

    def __del__(self, rmtree=shutil.rmtree):
        rmtree(self.folder, ignore_errors=True)


def prepare(case, seed):
    kind, state, seed = case["kind"], dict(case), seed % (1 << 25)
    if kind == "many":
        n, lo, hi = case["files"], case["low"], case["high"]
        state["inputs"] = []
        for i in range(n):  # spread evenly over the logarithm of the range, not in the order of size
            size = int(lo * (hi / lo) ** (((i * 2) % n + (2 * i >= n) * (1 - n % 2)) / max(n - 1, 1)))
            state["inputs"].append(_resident("gex" if i % 2 else "atac", size, seed * 64 + i, mixed=True))
        return state
    shape = case["shape"]
    if kind == "compress":  # whole blocks of records in an order of the seed's own
        n = int(case["bytes"] / RECORD[shape][0] * 1.02) + 2
        k = max(1, -(-n // UNIT_RECORDS))
        _, _, records, _ = _base_records(shape, n // k)
        data = torch.frombuffer(bytearray(records), dtype=torch.uint8).cuda().repeat(k)
        whole = case["bytes"] // bgzf.BLOCK_DATA
        order = torch.from_numpy(np.random.RandomState(seed).permutation(whole)).cuda()
        blocks = data[: whole * bgzf.BLOCK_DATA].view(whole, bgzf.BLOCK_DATA)[order].flatten()
        state["input"] = torch.cat([blocks, data[whole * bgzf.BLOCK_DATA : case["bytes"]]])
        return state
    if kind == "read":
        state["file"] = _File(_bam(shape, case["records"], seed)[1])
        return state
    comp, header = _resident(shape, case["records"], seed)
    if kind == "resident":
        state["input"] = comp, header
    elif kind == "plan":
        state["plan"] = batch.BatchPlan([(comp, header)], tags=TAGS[shape], form=0)
        state["plan"].capture()
    else:
        d = batch.decode_resident(comp, header, tags=())
        state["input"] = d.data.clone(), d.offset.clone(), header
    return state


# ---------------------------------------------------------------- calls


_SIGNED = {torch.uint16: torch.int16, torch.uint64: torch.int64}


def _whole(t):
    """A tensor of a type that every torch operation takes (the same bits)."""
    return t.view(_SIGNED[t.dtype]) if t.dtype in _SIGNED else t


def _tag(t):
    return {"type": t.type, "offset": t.offset, "length": t.length, "value": t.value}


def _columns(d):
    return {k: _whole(d.columns[k]) for k in FIELDS}


def _records(d):
    return {"data": d.data, "offset": d.offset, **_columns(d)}


def _file(d):
    return {**_records(d), "tags": {k: _tag(t) for k, t in d.tags.items()}}


def run(state):
    kind = state["kind"]
    if kind == "resident":
        comp, header = state["input"]
        return _file(batch.decode_resident(comp, header, tags=TAGS[state["shape"]]))
    if kind == "many":
        files = batch.decode_many(state["inputs"], tags=("CB", "UB"))
        return [{"data": d.data, "offset": d.offset, **{k: d.columns[k] for k in ("ref", "pos", "end", "mapq")},
                 "cb": d.tags["CB"].offset, "ub": d.tags["UB"].length} for d in files]
    if kind == "plan":
        return _file(state["plan"].replay()[0])
    if kind == "read":
        parts = []
        for b in cubam_b200.read_bam(state["file"].path, chunk_bytes=state["chunk"] or None):
            tags = b.tags(*TAGS[state["shape"]])
            parts.append({**_columns(b), "name": _whole(b.name_hash()), "cb": _whole(tags[0].hash()),
                          "type": tags[-1].type, "length": tags[-1].length})
        return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    if kind == "records":
        data, offset, header = state["input"]
        b = RecordBatch.decode(data, offset, header, derived=True)
        tags = b.tags(*TAGS[state["shape"]])
        codes, fits = tags[0].packed()
        last, names = tags[-1].strings(), b.names()
        return {**_records(b), "tags": [_tag(t) for t in tags], "codes": _whole(codes), "fits": fits, "hash": _whole(tags[-1].hash()),
                "strings": [last.chars, last.offsets], "names": [names.chars, names.offsets],
                "name_hash": _whole(b.name_hash()), "aligned": b.aligned_length(), "blocks": list(b.blocks()),
                "five_prime": b.five_prime(), "sizes": b.record_sizes()}
    return list(bgzf._bgzf_compress(state["input"], state["level"], return_offsets=True))


# ---------------------------------------------------------------- the bytes of a call


def _decode_bytes(shape, n, inflate=True):
    """Compressed bytes in (or the records' bytes, already inflated), inflated bytes, columns and tags out."""
    inflated, compressed = RECORD[shape]
    return n * (inflated + (compressed if inflate else 0) + COLUMN_BYTES + TAG_BYTES * len(TAGS[shape]))


def work(case):
    kind = case["kind"]
    if kind == "many":
        n, lo, hi = case["files"], case["low"], case["high"]
        sizes = [lo * (hi / lo) ** (i / max(n - 1, 1)) for i in range(n)]
        return {"bytes": sum(_decode_bytes("gex" if i % 2 else "atac", s) for i, s in enumerate(sizes)), "flops": 0}
    shape = case["shape"]
    if kind == "compress":
        return {"bytes": case["bytes"] * (1 + RECORD[shape][1] / RECORD[shape][0]), "flops": 0}
    n = case["records"]
    if kind == "records":
        # also codes, hashes, lengths, blocks, sizes, and two string columns (16-character names)
        return {"bytes": _decode_bytes(shape, n, inflate=False) + n * (9 + 8 + 8 + 4 + 16 + 4 + 8 + 2 * (16 + 4)), "flops": 0}
    return {"bytes": _decode_bytes(shape, n), "flops": 0}
