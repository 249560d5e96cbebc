"""Readers of one codec hand their page-locked buffers on: readers one after
another, several open at once with their batches interleaved, readers closed
half way, after an error, and after their codec -- each reads its own file."""

import threading

import numpy as np
import pytest

from fritillaria_gb300 import synth

pytestmark = pytest.mark.gpu


def _files(n):
    return [synth.short_read_bam(6000 + 500 * k, seed=k, levels=(1, 6)) for k in range(n)]


def _drain(reader):
    """The reader's whole output (no carry: members are read once)."""
    return np.concatenate([b.data.to_host() for b in reader])


@pytest.mark.parametrize("blocks", [1, 7, 300])
def test_readers_share_buffers(gpu, blocks):
    files = _files(4)
    codec = gpu.CudaCodec(0)
    for raw, bgzf in files + files[::-1]:
        assert np.array_equal(_drain(gpu.DeviceBgzfReader(bgzf, codec, blocks)), raw)
    # several at once, a batch each in turn
    readers = [gpu.DeviceBgzfReader(b, codec, blocks) for _, b in files]
    got = [[] for _ in files]
    live = set(range(len(files)))
    while live:
        for k in sorted(live):
            batch = readers[k].next_batch()
            if batch is None:
                live.discard(k)
            else:
                got[k].append(batch.data.to_host())
    for k, (raw, _) in enumerate(files):
        assert np.array_equal(np.concatenate(got[k]), raw)
    # one that failed, one left half way, then a whole one
    bad = files[0][1].copy()
    bad[len(bad) // 2] ^= 0x55
    with pytest.raises(gpu.FrtError):
        _drain(gpu.DeviceBgzfReader(bad, codec, blocks))
    half = gpu.DeviceBgzfReader(files[1][1], codec, blocks)
    half.next_batch()
    del half
    assert np.array_equal(_drain(gpu.DeviceBgzfReader(files[2][1], codec, blocks)), files[2][0])


def test_readers_of_one_codec_on_threads(gpu):
    files = _files(3)
    codec = gpu.CudaCodec(0)
    wrong = []

    def work(k):
        raw, bgzf = files[k]
        for _ in range(4):
            if not np.array_equal(_drain(gpu.DeviceBgzfReader(bgzf, codec, 5)), raw):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(files))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
