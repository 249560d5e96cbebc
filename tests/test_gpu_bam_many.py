"""The record stage over many short members, which a warp each scans: it does not
cost much more than the same bytes in full members (a CTA each took 4.5 times
as long)."""

import numpy as np
import pytest

from fritillaria_gb300 import synth

pytestmark = pytest.mark.gpu


def test_many_short_members_cost_little_more(gpu):
    torch = pytest.importorskip("torch")
    raw, ends = synth.raw_bam("short_reads", 130_000, seed=4)
    took, pos = {}, {}
    for payload in (1000, 65_280):
        bgzf = synth.bgzf(raw, "full", (1, 1), member_payload=payload)
        dev = torch.from_numpy(bgzf).to("cuda")
        torch.cuda.synchronize()
        eng = gpu.BatchEngine(0)
        eng.bind_bam(dev.data_ptr(), dev.numel())
        took[payload] = min(eng.time_stages(3)[2] for _ in range(3))
        eng.run()
        assert eng.finish().records == len(ends) - 1
        pos[payload] = eng.column("pos")
    assert np.array_equal(pos[1000], pos[65_280])
    assert took[1000] < 3 * took[65_280]


def test_offsets_past_the_batch_reach_no_byte_past_it(gpu):
    """Members that end up to 64 KiB past the batch are refused; the scan that
    runs before the refusal stays inside the batch, its prefetches too."""
    torch = pytest.importorskip("torch")
    raw, _ = synth.raw_bam("short_reads", 400, seed=5)
    dev = torch.from_numpy(raw).to("cuda")
    out = torch.zeros(1000, dtype=torch.int64, device="cuda")
    for offsets in ([0, 65_000, 65_000 + 60_000], [65_000, 130_000], [70_000, 10]):
        offs = torch.tensor(offsets, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        with pytest.raises(gpu.InvalidArgument):
            gpu.bam_scan_noalloc(dev.data_ptr(), 70_000, offs.data_ptr(), len(offsets) - 1, 0, out.data_ptr(), 1000, n_ref=1)
