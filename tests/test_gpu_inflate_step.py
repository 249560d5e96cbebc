"""Streams whose codes do not fall into step (2, 4, ... 256 equally likely
symbols: codes of one length, or nearly): the bytes zlib gives back, and no
longer than the serial form takes where the GPU is full."""

import struct
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [200, 3000, 24_000, 65_280, 65_536]


def _deflate(raw, level=6, strategy=zlib.Z_DEFAULT_STRATEGY):
    co = zlib.compressobj(level, zlib.DEFLATED, -15, 8, strategy)
    return co.compress(raw) + co.flush()


@pytest.mark.parametrize("symbols", [2, 4, 8, 16, 31, 32, 33, 64, 65, 127, 128, 129, 192, 250])
def test_equally_likely_symbols(gpu, symbols):
    from fritillaria_gb300 import SPAN_DTYPE

    rng = np.random.default_rng(symbols)
    data, spans, raws = bytearray(), [], []
    for n in SIZES:
        plain = rng.integers(0, symbols, n, dtype=np.uint8)
        far = plain.copy()  # now and then a match, its extra bits over a boundary
        for at in range(9000, n - 300, 1700):
            far[at:at + 7 + at % 250] = far[at - 8500:at - 8500 + 7 + at % 250]
        odd = plain.copy()  # and a symbol with a long code
        odd[::997] = 255
        for raw in (plain, far, odd):
            for level, strategy in ((1, 0), (6, 0), (6, zlib.Z_HUFFMAN_ONLY)):
                d = _deflate(raw.tobytes(), level, strategy)
                spans.append((len(data), len(data), len(d), n, zlib.crc32(raw.tobytes())))
                data += d + b"\xaa" * (8 + len(spans) % 4)
                raws.append(raw)
    got, offs = gpu.CudaCodec(0).inflate_batch(np.frombuffer(bytes(data), np.uint8), np.array(spans, dtype=SPAN_DTYPE))
    for i, raw in enumerate(raws):
        assert np.array_equal(got[offs[i]:offs[i + 1]], raw), i


@pytest.mark.parametrize("symbols", [64, 128])
@pytest.mark.parametrize("strategy", [zlib.Z_DEFAULT_STRATEGY, zlib.Z_HUFFMAN_ONLY])
def test_full_gpu_takes_no_longer_than_serial(gpu, symbols, strategy):
    """3,000 members, ten a CTA: the default took up to 2.3 times the serial
    form's time."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(symbols)
    head = b"BAM\x01" + struct.pack("<II", 0, 1) + struct.pack("<I", 5) + b"chr1\0" + struct.pack("<I", 1 << 28)
    raws = [head]
    for _ in range(20):  # a record a member: bases and qualities of any bytes
        bases, quals = rng.integers(0, symbols, 21_500, dtype=np.uint8).tobytes(), rng.integers(0, symbols, 43_000, dtype=np.uint8).tobytes()
        body = struct.pack("<iiBBHHHIiii", 0, 5, 2, 9, 0, 0, 4, 43_000, -1, -1, 0) + b"q\0" + bases + quals
        raws.append(struct.pack("<I", len(body)) + body)
    blocks = []
    for raw in raws:
        d = _deflate(raw, 6, strategy)
        blocks.append(b"\x1f\x8b\x08\x04\0\0\0\0\0\xff\x06\0BC\x02\0" + struct.pack("<H", len(d) + 25) + d + struct.pack("<II", zlib.crc32(raw), len(raw)))
    bgzf = np.frombuffer(blocks[0] + b"".join(blocks[1:]) * 150, np.uint8)
    dev = torch.from_numpy(bgzf.copy()).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1), reps=5)[0]
    serial = eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0]
    assert team < 1.1 * serial
    eng.run()
    assert eng.finish().status == 0
    assert eng.inflated().tobytes() == raws[0] + b"".join(raws[1:]) * 150
