"""The result sets a server adds for clients that hold their results are bounded and given back: past the bound a
batch waits for a release (an endless wait that nothing can end says so after a while), and a server whose clients
hold everything still closes."""
from __future__ import annotations

import time

import numpy as np
import pytest

from hpgbwt import lib, synth

pytestmark = pytest.mark.gpu

_ADDED = 256 << 20  # what the added sets may take


@pytest.fixture(scope="module")
def copies(tmp_path_factory):
    """Reads of 150 near-identical copies: dozens of hits and hundreds of rows each."""
    rng = np.random.default_rng(8)
    g = synth.genome("iid", 60_000, 45)
    elem = rng.integers(0, 4, 300, dtype=np.uint8)
    for k in range(150):
        cp = elem.copy()
        m = rng.random(300) < 0.02
        cp[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
        g[12_000 + k * 300: 12_000 + (k + 1) * 300] = cp
    d = tmp_path_factory.mktemp("copies")
    synth.write_fasta(str(d / "g.fa"), g, [30_000, 30_000])
    lib.build_index(str(d / "g.fa"), str(d / "idx"), 16)
    return g, str(d / "idx")


def _hold_until_stalled(srv, reads, per):
    """Requests submitted and waited for one by one, none released, until one is not published."""
    held = []
    for _ in range(2 * _ADDED // per + 8):
        t = srv.submit(reads.seq, reads.offsets)
        rs, _lat = srv.wait(t, timeout_ms=3000, copy=False)
        if rs is None:
            return held, t
        held.append(t)
    raise AssertionError(f"{len(held)} batches' results held ({len(held) * per >> 20} MB), still one more set added")


def test_added_sets_are_bounded_and_given_back(copies):
    g0, index = copies
    reads = synth.reads(g0, 4000, 9, length=(30, 60), edits="mix_30_50_20")
    with lib.GpuIndex(index) as g:
        want = g.search(reads, form=lib.FORM_BATCHED)
        per = want.hits.nbytes + want.locs.nbytes
        with lib.Server(g, max_batch_reads=4096) as srv:
            srv.wait(srv.submit(reads.seq, reads.offsets))
            held, stuck = _hold_until_stalled(srv, reads, per)
            assert len(held) >= 4
            starting = 3 * 1.5 * per + 3 * 4096 * 2 * 80 + (1 << 20)  # (starting sets grow by halves)
            assert srv.stats()["result_bytes"] <= _ADDED + starting
            t0 = time.time()
            with pytest.raises(RuntimeError, match="held by requests"):
                srv.wait(stuck)
            assert time.time() - t0 < 30
            queued = srv.submit(reads.seq, reads.offsets)
            with pytest.raises(RuntimeError, match="held by requests"):
                srv.wait(queued)
            assert srv.stats()["queued"] == 0  # its reads are the client's again
            srv.release(queued)
            srv.release(held.pop())
            rs, _lat = srv.wait(stuck, copy=False)  # the ticket was left as it was
            assert lib.result_from_c(rs, len(reads)).equal(want)
            for t in held + [stuck]:
                srv.release(t)
            until = time.time() + 20
            while srv.stats()["result_bytes"] > starting and time.time() < until:
                time.sleep(0.05)
                srv.wait(srv.submit(reads.seq, reads.offsets))
            assert srv.stats()["result_bytes"] <= starting
            res, _lat = srv.wait(srv.submit(reads.seq, reads.offsets))
            assert res.equal(want)


def test_server_closes_while_everything_is_held(copies):
    g0, index = copies
    reads = synth.reads(g0, 4000, 9, length=(30, 60), edits="mix_30_50_20")
    with lib.GpuIndex(index) as g:
        want = g.search(reads, form=lib.FORM_BATCHED)
        srv = lib.Server(g, max_batch_reads=4096)
        srv.wait(srv.submit(reads.seq, reads.offsets))
        _hold_until_stalled(srv, reads, want.hits.nbytes + want.locs.nbytes)
        srv.close()
        assert g.search(reads, form=lib.FORM_BATCHED).equal(want)
