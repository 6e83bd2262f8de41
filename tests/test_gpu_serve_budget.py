"""A server's admission counts what a batch holds: with reads of one hit and one row each, most of it are the offsets,
lists and queues of the reads themselves, some 400 bytes a read."""
from __future__ import annotations

import pytest

from hpgbwt import lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget_mb,alone", [(45, True), (400, False)])
def test_admission_counts_queues_and_lists(case_factory, budget_mb, alone):
    c = case_factory("iid", 200_000, 9, 2)
    warm = synth.reads(c.genome, 1024, 5, length=50)
    reqs = [synth.reads(c.genome, 60_000, 20 + i, length=50) for i in range(8)]
    with lib.GpuIndex(c.index) as g:
        with lib.Server(g, max_batch_reads=1 << 19, hbm_budget=budget_mb << 20) as srv:
            for _ in range(30):  # the server's estimates of hits and rows a read settle near one
                srv.wait(srv.submit(warm.seq, warm.offsets))
            st = srv.stats()
            assert st["hits_per_read"] < 1.2 and st["rows_per_read"] < 1.3
            got = [srv.wait(t)[0] for t in [srv.submit(r.seq, r.offsets) for r in reqs]]
            st = srv.stats()
        # one request holds 60000 x (400 + 80 a hit + 32 a row) + 1.25 bytes a base: some 36 MB
        assert st["max_batch_requests"] == 1 if alone else st["max_batch_requests"] > 1
        assert got[3].equal(g.search(reqs[3], form=lib.FORM_BATCHED))
