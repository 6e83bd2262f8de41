"""A client may hold any number of finished requests before it releases one: batches that find every result
set held get new ones, whatever order the client waits in."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("held", [2, 9])
def test_results_held_across_batches(case_factory, held):
    c = case_factory("repeats", 300_000, 3, 3)
    reqs = [synth.reads(c.genome, 200 + 10 * i, 700 + i, length=(36, 120), edits="mix_30_50_20") for i in range(held)]
    with lib.GpuIndex(c.index) as g:
        alone = [g.search(r, form=lib.FORM_BATCHED) for r in reqs]
        with lib.Server(g, max_batch_reads=4096) as srv:
            views = []
            for r in reqs:  # each waited for before the next is sent: a batch, and a result set, of its own
                t = srv.submit(r.seq, r.offsets)
                rs, _ = srv.wait(t, timeout_ms=20_000, copy=False)
                assert rs is not None, "the batch was never published"
                views.append((t, rs, len(r)))
            for (t, rs, n), want in zip(views, alone):
                assert lib.result_from_c(rs, n).equal(want)
                srv.release(t)
            assert srv.stats()["batches"] == held
