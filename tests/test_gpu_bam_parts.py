"""Record scans whose chains cross the eighths of a member that warps search and
walk apart: records of every size around a part (8,186 bytes of a full member),
records over many parts, members that hold no start, and names and payloads
that look like record headers where a part begins."""

import struct

import numpy as np
import pytest

from fritillaria_gb300 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def _record(size: int, decoys: bool, rng) -> bytes:
    """A record of `size` bytes in all: a name, no CIGAR or bases, one B:C array
    as filler, of record-like bytes if `decoys`."""
    name = b"q\0"
    fill = size - 36 - len(name) - 8
    assert fill >= 0
    fake = struct.pack("<iiiBBHHHIiii", 40, 0, 5, 2, 9, 0, 0, 0, 0, 0, 7, 0) + b"x\0" + bytes(4)
    body = (fake * (fill // len(fake) + 1))[:fill] if decoys else bytes(rng.integers(0, 256, fill, dtype=np.uint8))
    aux = b"XXBC" + struct.pack("<I", fill) + body
    core = struct.pack("<iiBBHHHIiii", 0, 5, len(name), 9, 0, 0, 0, 0, -1, -1, 0)
    return struct.pack("<I", size - 4) + core + name + aux


SIZES = {"short": (46, 330), "part": (8100, 8300), "parts": (9000, 70_000), "long": (60_000, 300_000), "smallest": (46, 47)}


@pytest.mark.parametrize("decoys", [False, True])
@pytest.mark.parametrize("shape", sorted(SIZES))
@pytest.mark.parametrize("payload", [65495, 8192, 1000])
def test_chains_over_parts(gpu, shape, decoys, payload):
    rng = np.random.default_rng(len(shape) + payload)
    lo, hi = SIZES[shape]
    text = b"@HD\tVN:1.6\n"
    head = b"BAM\x01" + struct.pack("<I", len(text)) + text + struct.pack("<I", 1) + struct.pack("<I", 5) + b"chr1\0" + struct.pack("<I", 1 << 28)
    parts, total = [head], len(head)
    while total < 400_000:
        r = _record(int(rng.integers(lo, hi)), decoys, rng)
        parts.append(r)
        total += len(r)
    raw = np.frombuffer(b"".join(parts), np.uint8)
    bgzf = synth.bgzf(raw, "full", (1, 1), member_payload=payload)
    want = oracle.decode_bam_file(bgzf)
    torch = pytest.importorskip("torch")
    dev = torch.from_numpy(np.ascontiguousarray(bgzf)).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    eng.run()
    st = eng.finish()
    assert st.records == len(want["columns"]["pos"]) == len(parts) - 1
    for k in ("record_offsets", "record_end", "aux_count", "aux_start"):
        assert np.array_equal(eng.column(k), want["columns"][k]), k
