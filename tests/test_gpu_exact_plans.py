"""The exact search's plans keep to themselves: a batch of short reads, thousands of rows each, leaves the plans of
the 1-error search at their size, and a server started later holds no plan of the exact search."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth
from oracle.pyoracle import PortOracle

pytestmark = pytest.mark.gpu


def _free() -> int:
    import torch
    return torch.cuda.mem_get_info()[0]


def test_rows_of_exact_batches_do_not_size_other_plans(case_factory):
    pytest.importorskip("torch")
    c = case_factory("iid", 200_000, 9, 2)
    rng = np.random.default_rng(2)
    short = synth.from_strings([bytes(rng.choice(list(b"ACGT"), 3).astype(np.uint8)) for _ in range(4000)])
    reads = synth.reads(c.genome, 70_000, 4, length=50, edits="mix_30_50_20")
    with lib.GpuIndex(c.index) as g:
        assert g.full_rows()
        got = g.search(short, mode=lib.MODE_EXACT, form=lib.FORM_BATCHED)
        rate = len(got.locs) / len(short)
        assert rate > 2000
        assert got.equal(g.search(short, mode=lib.MODE_EXACT, form=lib.FORM_PLAIN))
        before = _free()
        res = g.search(reads, mode=lib.MODE_SEARCH1, form=lib.FORM_BATCHED)
        took = before - _free()
        # at the exact batch's rate the locate pool alone of its 131072-read class
        assert took < 131072 * rate * 32 / 8
        with lib.Server(g, max_batch_reads=4096) as srv:
            t = srv.submit(reads.seq[:int(reads.offsets[100])], reads.offsets[:101])
            srv.wait(t)
            assert srv.stats()["plan_bytes"] < 4096 * rate * 32 * 4
        assert g.search(short, mode=lib.MODE_EXACT, form=lib.FORM_BATCHED).equal(got)
    want = PortOracle(c.index).search(reads, mode=lib.MODE_SEARCH1, max_results=1 << 16, threads=8)
    assert res.equal(want)
