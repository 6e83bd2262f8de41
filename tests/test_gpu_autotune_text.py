"""The autotuner with the whole suffix arrays in use: settings that the search with the text does not read are
neither timed apart, nor changed by the noise between equal runs, nor paid for with a start table."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth

pytestmark = pytest.mark.gpu


def test_settings_without_effect_stay(case_factory):
    torch = pytest.importorskip("torch")
    c = case_factory("iid", 1_000_000, 33, 1)
    reads = synth.reads(c.genome, 40_000, 39, length=(80, 150), edits="mix_30_50_20")
    d_seq = torch.from_numpy(reads.seq).cuda()
    d_off = torch.from_numpy(reads.offsets.view(np.int64)).cuda()
    args = (d_seq.data_ptr(), d_off.data_ptr(), len(reads), int(reads.offsets[-1]),
            int(np.diff(reads.offsets).max()), 64)
    with lib.GpuIndex(c.index) as g:
        g.set_wave_group(32)
        g.set_direction_split(0)
        want = g.search(reads, form=lib.FORM_BATCHED, max_results=64)
        table = g.autotune(*args)
        warp = [r["search_us"] for r in table if r["stack"] == -2][:12]
        assert len(set(warp)) == 1 and warp[0] < min(r["search_us"] for r in table[:60])
        assert g.wave_group() == 32 and g.direction_split() == 0 and g.start_table() == 0
        assert g.search(reads, form=lib.FORM_BATCHED, max_results=64).equal(want)
        g.set_full_rows(False)  # without the arrays they are settings again
        table = g.autotune(*args)
        assert len({r["search_us"] for r in table if r["stack"] == -2}) > 1
        assert g.search(reads, form=lib.FORM_BATCHED, max_results=64).equal(want)
