"""A program that wants the device's memory gets back what the whole suffix arrays and the text take, and every call
goes on with the sampled arrays, with the same results."""
from __future__ import annotations

import pytest

from hpgbwt import lib, synth

pytestmark = pytest.mark.gpu


def test_dropped_arrays_give_their_memory_back(case_factory):
    torch = pytest.importorskip("torch")
    c = case_factory("repeats", 4_000_000, 21, 2)
    reads = synth.reads(c.genome, 3000, 6, length=(36, 150), edits="mix_30_50_20")
    with lib.GpuIndex(c.index) as g:
        assert g.full_rows()
        calls = {
            "batched": lambda: g.search(reads, form=lib.FORM_BATCHED),
            "plain": lambda: g.search(reads, form=lib.FORM_PLAIN),
            "exact": lambda: g.search(reads, mode=lib.MODE_EXACT, form=lib.FORM_BATCHED),
            "block": lambda: g.block_search(reads, max_results=64),
        }
        want = {k: f() for k, f in calls.items()}
        before = torch.cuda.mem_get_info()[0]
        g.drop_full_rows()
        assert torch.cuda.mem_get_info()[0] - before >= 16 * 4_000_000
        assert not g.full_rows() and not g.set_full_rows(True)
        for k, f in calls.items():
            assert f().equal(want[k]), k
            assert f().equal(want[k]), f"{k}, again"
        g.drop_full_rows()  # nothing left to give back
        with lib.Server(g, max_batch_reads=4096) as srv:
            assert srv.wait(srv.submit(reads.seq, reads.offsets))[0].equal(want["batched"])
