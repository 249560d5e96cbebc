"""Launches of many members, short ones among them or all of them short, where a
warp a member is quicker than a team: the bytes zlib gives back, the oracle's
error for a bad member among them, and no longer than the serial form takes."""

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _file(streams):
    """The streams back to back at odd distances, and their spans."""
    from fritillaria_gb300 import SPAN_DTYPE

    data, spans = bytearray(b"\x55" * 3), []
    for k, (payload, raw) in enumerate(streams):
        spans.append((len(data), len(data), len(payload), len(raw), zlib.crc32(raw)))
        data += payload + b"\xaa" * (8 + k % 5)
    return np.frombuffer(bytes(data), np.uint8), np.array(spans, dtype=SPAN_DTYPE)


def _deflate(raw, level=6, strategy=zlib.Z_DEFAULT_STRATEGY, mem=8):
    co = zlib.compressobj(level, zlib.DEFLATED, -15, mem, strategy)
    return co.compress(raw) + co.flush()


def _streams(n, rng):
    """Members of 0 to 4,000 bytes (n odd) or 500, one in 50 long (n even);
    text and runs, every level."""
    letters = np.frombuffer(b"ACGTNacgt\t\n0123456789", np.uint8)
    out = []
    for k in range(n):
        size = int(rng.integers(0, 4000 if n % 2 else 500)) if n % 2 or k % 50 else int(rng.integers(30_000, 65_537))
        raw = bytes(rng.choice(letters, size)) if k % 3 else bytes(letters[:7]) * (size // 7)
        out.append((_deflate(raw, int(rng.integers(0, 10))), raw))
    return out


@pytest.mark.parametrize("n", [1, 303, 305, 607, 608, 913, 2500, 2501, 5000, 5001])
def test_many_members_equal_zlib(gpu, n):
    """Counts around one, two, three and many members a CTA of a 152-SM grid."""
    streams = _streams(n, np.random.default_rng(n))
    data, spans = _file(streams)
    got, offs = gpu.CudaCodec(0).inflate_batch(data, spans)
    for i, (_, raw) in enumerate(streams):
        assert got[offs[i]:offs[i + 1]].tobytes() == raw, i


@pytest.mark.parametrize("bad", [0, 1500, 2999])
def test_a_bad_member_among_short_ones(gpu, bad):
    from oracle import oracle

    streams = [(_deflate(b"a%d" % k * 40), b"a%d" % k * 40) for k in range(3000)]
    payload, raw = streams[bad]
    streams[bad] = (payload[:-3], raw)
    data, spans = _file(streams)
    with pytest.raises(oracle.OracleError) as oe:
        oracle.inflate_batch(data, spans)
    with pytest.raises(gpu.FrtError) as ge:
        gpu.CudaCodec(0).inflate_batch_device(data, spans)
    assert (ge.value.code, ge.value.offset) == (oe.value.code, oe.value.offset)


@pytest.mark.parametrize("payload", [400, 1000])
def test_short_members_take_no_longer_than_serial(gpu, payload):
    """20,000 members and over, each a few records: the default took two to three
    times the serial form's time where every member had a team."""
    torch = pytest.importorskip("torch")
    from fritillaria_gb300 import synth

    raw, bgzf = synth.short_read_bam(20_000 * payload // 296, seed=9, member_payload=payload)
    dev = torch.from_numpy(bgzf).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    team = eng.time_inflate(gpu.InflateTuning(0, 3, 0, 1), reps=5)[0]
    serial = eng.time_inflate(gpu.InflateTuning(1, 3, 0, 1), reps=5)[0]
    assert team < 1.3 * serial
    eng.run()
    assert eng.finish().status == 0 and np.array_equal(eng.inflated(), raw)
