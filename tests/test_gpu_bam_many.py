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
