"""Chunks of up to 4,096 and 8,192 bytes, which are compressed several to an SM
where there are many: the same block as alone, zlib's bytes back, in batches of
one length and of mixed ones; and 5,000 short chunks take no longer than a few
times 100 of them (one an SM, they took 18 times as long)."""

import time
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bytes(n, rng):
    """Text with matches of many lengths and distances, noise between."""
    out = [rng.choice(np.frombuffer(b"ACGTN\t0123456789", np.uint8), 600)]
    size = 600
    while size < n:
        k = int(rng.integers(3, 300))
        if rng.random() < 0.6:
            done = np.concatenate(out) if len(out) > 1 else out[0]
            out = [done]
            at = int(rng.integers(0, size - 1))
            piece = np.resize(done[at:at + k], k)
        else:
            piece = rng.integers(0, 256, k % 40 + 1, dtype=np.uint8)
        out.append(piece)
        size += piece.size
    return np.concatenate(out)[:n]


def _check(gpu, data, bounds, alone):
    torch = pytest.importorskip("torch")
    dev = torch.from_numpy(data).to("cuda")
    torch.cuda.synchronize()
    comp = gpu.DeviceCompressor(0)
    bounds = np.asarray(bounds, np.uint64)
    got = comp.compress_batch_device(dev.data_ptr(), dev.numel(), bounds)
    for i in range(len(bounds) - 1):
        raw, block = data[int(bounds[i]):int(bounds[i + 1])].tobytes(), got.block(i).tobytes()
        assert zlib.decompress(block[18:-8], -15) == raw, i
        assert int.from_bytes(block[-8:-4], "little") == zlib.crc32(raw) and int.from_bytes(block[-4:], "little") == len(raw)
        if i in alone:
            assert comp.compress_batch_device(dev.data_ptr(), dev.numel(), bounds[i:i + 2]).block(0).tobytes() == block, i


@pytest.mark.parametrize("size,count", [(1, 700), (33, 700), (513, 1500), (4095, 700), (4096, 700), (4096, 300), (4097, 300), (8191, 300), (8192, 300), (8193, 160)])
def test_many_chunks_of_one_length(gpu, size, count):
    data = _bytes(size * count, np.random.default_rng(size))
    _check(gpu, data, np.arange(count + 1) * size, {0, 1, count // 2, count - 1})


@pytest.mark.parametrize("small,medium,large", [(700, 200, 20), (700, 3, 0), (200, 5, 1), (100, 100, 3), (0, 200, 1), (700, 0, 1)])
def test_chunks_of_mixed_lengths(gpu, small, medium, large):
    rng = np.random.default_rng(small + medium)
    sizes = np.concatenate([rng.integers(0, 4097, small), rng.integers(4097, 8193, medium), rng.integers(8193, 65_506, large)])
    rng.shuffle(sizes)
    bounds = np.concatenate([[0], np.cumsum(sizes)])
    _check(gpu, _bytes(int(bounds[-1]) + 1, rng), bounds, set(range(0, len(sizes), 50)))


def test_many_short_chunks_cost_little_more_than_few(gpu):
    torch = pytest.importorskip("torch")
    data = _bytes(200_000, np.random.default_rng(2))
    dev = torch.from_numpy(np.resize(data, 1_500_000)).to("cuda")
    torch.cuda.synchronize()
    comp = gpu.DeviceCompressor(0)
    out = np.empty(66_000 * 5000, np.uint8)
    took = {}
    for count in (100, 5000):
        bounds = np.arange(count + 1, dtype=np.uint64) * 300
        for _ in range(5):
            t = time.perf_counter()
            comp.compress_batch_device(dev.data_ptr(), dev.numel(), bounds, out)
            took[count] = min(took.get(count, 1.0), time.perf_counter() - t)
    assert took[5000] < 8 * took[100]


def _took(gpu, data, size, turns=5):
    torch = pytest.importorskip("torch")
    dev = torch.from_numpy(data).to("cuda")
    torch.cuda.synchronize()
    comp = gpu.DeviceCompressor(0)
    bounds = np.arange(0, data.size + 1, size, dtype=np.uint64)
    out = np.empty(66_000 * len(bounds), np.uint8)
    best = 1.0
    for _ in range(turns):
        t = time.perf_counter()
        comp.compress_batch_device(dev.data_ptr(), dev.numel(), bounds, out)
        best = min(best, time.perf_counter() - t)
    return best


def test_runs_cost_no_more_than_noise(gpu):
    """450 chunks of zeros, whose every position has a match of 258 bytes, against
    450 of noise, which has none (comparing each position alone, they took 1.3
    times as long)."""
    size = 65_280
    assert _took(gpu, np.zeros(450 * size, np.uint8), size) < _took(gpu, np.random.default_rng(1).integers(0, 256, 450 * size, dtype=np.uint8), size)


@pytest.mark.parametrize("period", [1, 2, 3, 4, 31, 32, 33, 63, 64, 65, 300, 5000])
def test_repeated_blocks_round_trip(gpu, period):
    """Runs of one distance, broken now and then by another byte or another period."""
    rng = np.random.default_rng(period)
    unit, other = rng.integers(0, 256, period, dtype=np.uint8), rng.integers(0, 4, 40, dtype=np.uint8)
    data = np.resize(unit, 200_000)
    at = rng.integers(0, data.size, 60)
    data[at] ^= 1
    for k in at[:20]:
        data[k:k + 400] = np.resize(other, 400)[:data[k:k + 400].size]
    sizes = [1, 31, 32, 33, 64, 300, 1000, 4096, 4097, 8192, 8193, 30_000, 65_505]
    _check(gpu, data, np.concatenate([[0], np.cumsum(sizes)]), set(range(len(sizes))))
