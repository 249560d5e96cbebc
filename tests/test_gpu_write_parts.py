"""The device deflate at the sizes where its parts meet: chunks around a step (32
positions), a thread's and a warp's share, the window, the largest payload, and
chunks whose length leaves some of the parsing warps nothing; runs,
matches across parts, long matches and noise.  zlib turns every block back into
its chunk, and the same chunk gives the same block alone and among others."""

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 31, 32, 33, 63, 64, 65, 511, 512, 513, 1023, 1025, 4093, 4095, 4097, 8191, 16_000, 32_767, 32_768, 32_771, 65_280, 65_504, 65_505]


def _content(kind: str, n: int, rng) -> np.ndarray:
    if kind == "zeros":
        return np.zeros(n, np.uint8)
    if kind == "bases":
        return rng.choice(np.frombuffer(b"ACGT", np.uint8), n)
    if kind == "noise":
        return rng.integers(0, 256, n, dtype=np.uint8)
    if kind == "far":  # matches at the window's edge: 32,768 back and one past it
        unit = rng.integers(0, 256, 32_768 + int(rng.integers(0, 2)), dtype=np.uint8)
        return np.resize(unit, n)
    unit = rng.integers(0, 256, 1000, dtype=np.uint8)  # "long": matches of every length up to 258 and over
    out = np.concatenate([np.concatenate([unit[: 3 + k % 300], rng.integers(0, 256, 1 + k % 3, dtype=np.uint8)]) for k in range(max(1, n // 100 + 1))])
    return np.resize(out, n)


@pytest.mark.parametrize("kind", ["zeros", "bases", "noise", "far", "long"])
def test_blocks_round_trip(gpu, kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(7)
    chunks = [_content(kind, n, rng) for n in SIZES]
    data = np.concatenate(chunks)
    bounds = np.concatenate([[0], np.cumsum([c.size for c in chunks])]).astype(np.uint64)
    dev = torch.from_numpy(data).to("cuda")
    torch.cuda.synchronize()
    comp = gpu.DeviceCompressor(0)
    got = comp.compress_batch_device(dev.data_ptr(), dev.numel(), bounds)
    for i, c in enumerate(chunks):
        block = got.block(i).tobytes()
        assert zlib.decompress(block[18:-8], -15) == c.tobytes(), (kind, c.size)
        assert int.from_bytes(block[-8:-4], "little") == zlib.crc32(c.tobytes()) and int.from_bytes(block[-4:], "little") == c.size
        one = comp.compress_batch_device(dev.data_ptr(), dev.numel(), bounds[i:i + 2])
        assert one.block(0).tobytes() == block, (kind, c.size)
