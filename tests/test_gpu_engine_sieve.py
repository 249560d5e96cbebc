"""Device member discovery where headers fall on the edges of the sieve's steps:
member starts at every distance around 16-byte lanes, 512-byte steps, 2 KiB
groups of loads and 8 KiB tiles, payloads full of the magic bytes, and buffers
that end anywhere in a tile."""

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _member(payload: bytes, size: int | None = None) -> bytes:
    """A stored member, its extra field padded to `size` bytes in all if given."""
    body = b"\x01" + len(payload).to_bytes(2, "little") + (len(payload) ^ 0xFFFF).to_bytes(2, "little") + payload
    pad = 0 if size is None else size - (18 + len(body) + 8)
    extra = b"BC\x02\x00%s"
    if pad:
        assert pad >= 4
        extra = b"XX" + (pad - 4).to_bytes(2, "little") + b"\x1f\x8b\x08\x04"[: pad - 4].ljust(pad - 4, b"\x1f") + extra
    total = 12 + len(extra) + len(body) + 8  # "%s" stands for the two size bytes
    head = b"\x1f\x8b\x08\x04\0\0\0\0\0\xff" + len(extra).to_bytes(2, "little") + extra.replace(b"%s", (total - 1).to_bytes(2, "little"))
    return head + body + zlib.crc32(payload).to_bytes(4, "little") + len(payload).to_bytes(4, "little")


@pytest.mark.parametrize("edge", [16, 512, 2048, 8192])
def test_headers_around_an_edge(gpu, edge):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(edge)
    blob, parts = b"", []
    for k in range(60):
        # the next member starts `back` bytes before a multiple of the edge
        back = k % 20
        target = (len(blob) // edge + 1 + (300 + edge) // edge) * edge - back
        payload = bytes(rng.choice(np.frombuffer(b"\x1f\x8b\x08\x04ACGT\n", np.uint8), int(rng.integers(1, 120))))
        blob += _member(payload, target - len(blob))
        assert len(blob) == target
        parts.append(payload)
    tail = bytes(rng.integers(65, 90, edge % 700 + 1, dtype=np.uint8))
    blob += _member(tail)
    parts.append(tail)
    data = np.frombuffer(blob, np.uint8)
    dev = torch.from_numpy(data.copy()).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_files(dev.data_ptr(), dev.numel(), [(0, dev.numel(), gpu.Format.FASTA)])
    eng.run()
    assert eng.finish().status == 0
    assert eng.file_info(0).members == len(parts)
    assert eng.inflated().tobytes() == b"".join(parts)
