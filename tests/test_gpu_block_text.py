"""The block search with the text on the device against the oracle and against rank steps: fragment edges, errors
at every position near them, repeats whose insertion goes on into a mismatch, capacities that cut the results."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth
from oracle.pyoracle import PortOracle

pytestmark = pytest.mark.gpu

_A = np.frombuffer(b"ACGT", dtype=np.uint8)


def _reads(g: np.ndarray, seed: int) -> synth.ReadSet:
    rng = np.random.default_rng(seed)
    out = []
    for L in (30, 59, 60, 61, 62, 63, 89, 90, 100, 121, 128, 160):
        frag = max(L // 2, 30)
        for p in (0, len(g) - L - 1, int(rng.integers(0, len(g) - L - 1)), int(rng.integers(0, len(g) - L - 1))):
            f = g[p:p + L + 1]
            for at in {0, 1, frag - 2, frag - 1, frag, frag + 1, L - 2, L - 1, int(rng.integers(0, L))}:
                at = min(max(at, 0), L - 1)
                sub = f[:L].copy()
                sub[at] = (sub[at] + rng.integers(1, 4)) % 4
                for r in (f[:L], sub, np.insert(f[:L - 1], at, rng.integers(0, 4)).astype(np.uint8), np.delete(f, at)):
                    out.append(_A[r if rng.random() < 0.5 else synth.revcomp_codes(r)].tobytes())
    return synth.from_strings(out)


@pytest.mark.parametrize("max_results", [1, 2, 1 << 16])
@pytest.mark.parametrize("kind,n", [("iid", 3000), ("human_like", 60_000)])
def test_block_search_with_text(case_factory, kind, n, max_results):
    c = case_factory(kind, n, 17, 2)
    reads = _reads(c.genome, 3)
    want = PortOracle(c.index).block_search(reads, max_results=max_results, threads=8)
    assert len(want.result.hits) > 1000
    with lib.GpuIndex(c.index) as g:
        for rows in (True, False):
            assert g.set_full_rows(rows) == rows
            assert g.block_search(reads, max_results=max_results).equal(want), f"full rows {rows}"
