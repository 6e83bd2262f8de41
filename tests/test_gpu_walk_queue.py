"""More one-row walks than the walk queue of the search with the text holds: the lanes that find it full go on by
rank steps, and no slot is read that nothing was written to, for read counts that leave the queue's end inside a
chunk of slots (the direct form takes the caller's read count; the captured one a power of two)."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth
from oracle.pyoracle import PortOracle

pytestmark = pytest.mark.gpu

_A = np.frombuffer(b"ACGT", dtype=np.uint8)


@pytest.fixture(scope="module")
def copies(tmp_path_factory):
    """1500 copies of one 220-base stretch, each with 2 % of its own substitutions: a read of 100 bases of one stays
    wide far into the branching window, loses a few rows at nearly every base there, and each base that other
    copies have in its place begins a walk of a row or two: some 45 that reach one row a read, for which the lanes ask
    3.7 million slots where the queue holds 2.8."""
    rng = np.random.default_rng(3)
    unit = rng.integers(0, 4, 220, dtype=np.uint8)
    g = np.tile(unit, 1500)
    m = rng.random(len(g)) < 0.02
    g[m] = rng.integers(0, 4, int(m.sum()), dtype=np.uint8)
    d = tmp_path_factory.mktemp("copies")
    synth.write_fasta(str(d / "g.fa"), g)
    lib.build_index(str(d / "g.fa"), str(d / "idx"), 16)
    return g, str(d / "idx")


@pytest.mark.parametrize("n", [80_000, 80_001, 80_003])
def test_full_walk_queue_matches_oracle(copies, n):
    g0, index = copies
    rng = np.random.default_rng(n)
    at = rng.integers(0, len(g0) - 100, n)
    reads = synth.from_strings([_A[g0[p:p + 100]].tobytes() for p in at])
    want = PortOracle(index).search(reads, mode=lib.MODE_SEARCH1, max_results=1 << 16, threads=8)
    with lib.GpuIndex(index) as g:
        assert g.full_rows()
        g.set_graph(False)
        assert g.search(reads, mode=lib.MODE_SEARCH1, form=lib.FORM_BATCHED).equal(want)
        if n & 1:
            g.set_graph(True)
            assert g.search(reads, mode=lib.MODE_SEARCH1, form=lib.FORM_BATCHED).equal(want)
