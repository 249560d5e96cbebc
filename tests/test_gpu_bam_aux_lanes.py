"""Aux strings a few lanes or all of a warp look through: lengths around the bytes
a lane takes alone (64 and 96 for each lane whose string goes on), ended,
unended and among short ones; and records of 100-byte strings cost no more than
those of short ones (their record stage took seven times as long)."""

import struct

import numpy as np
import pytest

from fritillaria_gb300 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

TEXT = b"@HD\tVN:1.6\n"
HEAD = b"BAM\x01" + struct.pack("<I", len(TEXT)) + TEXT + struct.pack("<I", 1) + struct.pack("<I", 5) + b"chr1\0" + struct.pack("<I", 1 << 28)


def _record(name: bytes, aux: bytes) -> bytes:
    body = struct.pack("<iiBBHHHIiii", 0, 5, len(name), 9, 0, 0, 0, 0, -1, -1, 0) + name + aux
    return struct.pack("<I", len(body)) + body


def _engine(gpu, bgzf):
    torch = pytest.importorskip("torch")
    dev = torch.from_numpy(np.ascontiguousarray(bgzf)).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    return eng, dev


@pytest.mark.parametrize("lanes", [1, 2, 13, 31, 32])
@pytest.mark.parametrize("ended", [True, False])
def test_lengths_around_the_handover(gpu, lanes, ended):
    rng = np.random.default_rng(lanes)
    out = [HEAD]
    for turn in range(6):
        for k in range(32):
            n = 64 + 96 * lanes + int(rng.integers(-40, 41)) if k < lanes else int(rng.integers(0, 30))
            value = bytes(rng.integers(33, 127, n, dtype=np.uint8))
            open_end = not ended and k == turn
            out.append(_record(b"q" * (1 + (k + turn) % 16) + b"\0", b"NMC\x05MMZ" + value + (b"" if open_end else b"\0XAc\x01")))
    bgzf = synth.bgzf(np.frombuffer(b"".join(out), np.uint8), "full", (1, 1))
    want = oracle.decode_bam_file(bgzf)
    eng, _ = _engine(gpu, bgzf)
    eng.run()
    assert eng.finish().records == len(out) - 1
    for k in ("aux_count", "aux_status"):
        assert np.array_equal(eng.column(k), want["columns"][k]), k
    got, cols = eng.column("aux_entries"), {k: eng.column(k) for k in ("record_offsets", "aux_start", "record_end", "aux_first")}
    for i, off in enumerate(cols["record_offsets"]):
        e, _ = oracle.bam_aux(want["inflated"], int(off), int(cols["aux_start"][i]), int(cols["record_end"][i]))
        assert np.array_equal(got[cols["aux_first"][i]:cols["aux_first"][i + 1]], e.astype(got.dtype)), i


def test_strings_of_every_record_cost_no_more(gpu):
    rng = np.random.default_rng(3)
    took = {}
    for n in (10, 100):
        parts, ends = [HEAD], [len(HEAD)]
        while ends[-1] < 60_000_000:
            z = rng.integers(33, 127, 2 * n, dtype=np.uint8).tobytes()
            chunk = _record(b"q\0", b"NMC\x05XAZ" + z[:n] + b"\0XBZ" + z[n:] + b"\0") * 500
            parts.append(chunk)
            ends.append(ends[-1] + len(chunk))
        eng, _ = _engine(gpu, synth.bgzf(np.frombuffer(b"".join(parts), np.uint8), "full", (1, 1)))
        took[n] = min(eng.time_stages(3)[2] for _ in range(3))
    assert took[100] < 2 * took[10]
