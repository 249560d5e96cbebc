"""Which form decodes a member: the streams of the team's edge test are all
decoded by the team, bad ones and members of short blocks in a full launch are
handed over, and a small launch's time is the team's, not the serial form's."""

import zlib

import numpy as np
import pytest
from test_gpu_inflate_team import SIZES, _content, _deflate, _file

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["zeros", "period", "pairs", "skewed", "noise", "mixed"])
def test_the_team_decodes_valid_members(gpu, kind):
    rng = np.random.default_rng(len(kind))
    streams = []
    for n in SIZES:
        raw = _content(kind, n, rng)
        for level, strategy, mem in ((1, 0, 8), (6, 0, 8), (9, 0, 1), (6, zlib.Z_HUFFMAN_ONLY, 8), (6, zlib.Z_FIXED, 9), (0, 0, 8)):
            streams.append((_deflate(raw, level, strategy, mem), raw))
    data, spans = _file(streams)
    before = gpu.inflate_handed_over()
    got, offs = gpu.CudaCodec(0).inflate_batch(data, spans)
    assert gpu.inflate_handed_over() == before
    for i, (_, raw) in enumerate(streams):
        assert got[offs[i]:offs[i + 1]].tobytes() == raw, (kind, i)


def test_bad_members_are_handed_over(gpu):
    raw = _content("mixed", 30_000, np.random.default_rng(1))
    d = _deflate(raw, 6)
    for bad in (d[:-5], d[:40], b"\x07" + d[1:]):  # cut in a block, in its header; a block of no type
        data, spans = _file([(d, raw), (bad, raw), (d, raw)])
        before = gpu.inflate_handed_over()
        with pytest.raises(gpu.InflateError):
            gpu.CudaCodec(0).inflate_batch_device(data, spans)
        assert gpu.inflate_handed_over() == before + 1


def test_short_blocks_are_handed_over_in_full_launches_only(gpu):
    rng = np.random.default_rng(2)
    text = rng.choice(np.frombuffer(b"ACGTN\t\n0123456789", np.uint8), 60_000).tobytes()
    stream = (_deflate(text, 6, 0, 1), text)
    for n, handed in ((200, False), (1500, True)):
        data, spans = _file([stream] * n)
        before = gpu.inflate_handed_over()
        got, _ = gpu.CudaCodec(0).inflate_batch(data, spans)
        assert got.tobytes() == text * n
        assert (gpu.inflate_handed_over() - before > n // 2) == handed


def test_a_small_launch_takes_the_teams_time(gpu):
    torch = pytest.importorskip("torch")
    from fritillaria_gb300 import synth

    _, bgzf = synth.short_read_bam(60_000, seed=6)
    dev = torch.from_numpy(bgzf).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1, spread_variant=1), reps=5)[0]
    assert team < eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0] / 4
