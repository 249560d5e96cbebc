"""Aux strings whose end is looked for by a lane alone, then by its warp: lengths
around the handover (64 bytes), 16-byte blocks, 512-byte and 2 KiB turns, at
every alignment, unterminated ones and H strings among them."""

import struct

import numpy as np
import pytest

from fritillaria_gb300 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 15, 16, 17, 62, 63, 64, 65, 66, 79, 80, 81, 127, 128, 500, 511, 512, 513, 2046, 2047, 2048, 2049, 2112, 2113, 4200, 20_000]


@pytest.mark.parametrize("shift", range(0, 16, 3))
@pytest.mark.parametrize("kind", ["Z", "H", "open"])
def test_string_ends(gpu, kind, shift):
    torch = pytest.importorskip("torch")
    text = b"@HD\tVN:1.6\n"
    out = [b"BAM\x01" + struct.pack("<I", len(text)) + text + struct.pack("<I", 1) + struct.pack("<I", 5) + b"chr1\0" + struct.pack("<I", 1 << 28)]
    rng = np.random.default_rng(shift)
    for n in LENGTHS * 2:
        name = b"q" * (1 + (shift + n) % 16) + b"\0"
        if kind == "H":
            n += n & 1
        letters = np.frombuffer(b"0123456789ABCDEFabcdef", np.uint8) if kind == "H" else np.arange(33, 127, dtype=np.uint8)
        value = bytes(rng.choice(letters, n))
        aux = b"NMC\x05" + b"MM" + (b"H" if kind == "H" else b"Z") + value + (b"" if kind == "open" else b"\0XAc\x01")
        body = struct.pack("<iiBBHHHIiii", 0, 5, len(name), 9, 0, 0, 0, 0, -1, -1, 0) + name + aux
        out.append(struct.pack("<I", len(body)) + body)
    bgzf = synth.bgzf(np.frombuffer(b"".join(out), np.uint8), "full", (1, 1))
    want = oracle.decode_bam_file(bgzf)
    dev = torch.from_numpy(np.ascontiguousarray(bgzf)).to("cuda")
    torch.cuda.synchronize()
    eng = gpu.BatchEngine(0)
    eng.bind_bam(dev.data_ptr(), dev.numel())
    eng.run()
    assert eng.finish().records == len(out) - 1
    for k in ("aux_count", "aux_status"):
        assert np.array_equal(eng.column(k), want["columns"][k]), k
    got, cols = eng.column("aux_entries"), {k: eng.column(k) for k in ("record_offsets", "aux_start", "record_end", "aux_first")}
    for i, off in enumerate(cols["record_offsets"]):
        e, _ = oracle.bam_aux(want["inflated"], int(off), int(cols["aux_start"][i]), int(cols["record_end"][i]))
        assert np.array_equal(got[cols["aux_first"][i]:cols["aux_first"][i + 1]], e.astype(got.dtype)), i
