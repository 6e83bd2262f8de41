"""Reads that leave a repeat of many exact copies, or a tandem run, for sequence that occurs once: chains too wide for
a lane per row, whose change points the strand's other chain decides where it can, against the oracle.  Errors near
the junction, near the head of the other chain and at the read's ends; both forms, both strands."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth
from oracle.pyoracle import PortOracle

pytestmark = pytest.mark.gpu

_A = np.frombuffer(b"ACGT", dtype=np.uint8)


def _genome(rng: np.random.Generator, unit: int) -> tuple[np.ndarray, np.ndarray, int]:
    """A random genome with 150 copies of one stretch (unit 0: 180 random bases, else a tandem run of `unit` bases),
    the copies' starts and their length."""
    g = rng.integers(0, 4, 150_000, dtype=np.uint8)
    n = 180
    copy = rng.integers(0, 4, n, dtype=np.uint8) if unit == 0 else \
        np.resize(np.arange(unit, dtype=np.uint8), n)
    at = 500 + 900 * np.arange(150)
    for s in at:
        g[s:s + n] = copy
    return g, at, n


def _reads(g, starts, n, rng) -> synth.ReadSet:
    out = []
    for L in (40, 64, 100, 151, 240):
        for share in (0.2, 0.45, 0.5, 0.55, 0.8, 0.95):
            inside = int(L * share)
            for s in rng.choice(starts, 6, replace=False):
                for p, junction in ((s + n - inside, inside), (s - (L - inside), L - inside)):
                    f = g[p:p + L + 1]
                    for at in {0, 1, junction - 2, junction - 1, junction, junction + 1, junction + 14,
                               L - 15, L - 14, L - 2, L - 1, int(rng.integers(0, L))}:
                        at = min(max(int(at), 0), L - 1)
                        sub = f[:L].copy()
                        sub[at] = (sub[at] + rng.integers(1, 4)) % 4
                        two = sub.copy()
                        other = int(rng.integers(0, L))
                        two[other] = (two[other] + 1) % 4
                        r = (f[:L], sub, two, np.insert(f[:L - 1], at, rng.integers(0, 4)).astype(np.uint8),
                             np.delete(f, at))[int(rng.integers(0, 5))]
                        out.append(_A[r if rng.random() < 0.5 else synth.revcomp_codes(r)].tobytes())
    return synth.from_strings(out)


@pytest.mark.parametrize("unit", [0, 1, 2, 3])
def test_wide_chains_match_oracle(tmp_path, unit):
    rng = np.random.default_rng(40 + unit)
    g0, starts, n = _genome(rng, unit)
    synth.write_fasta(str(tmp_path / "g.fa"), g0, [90_000, 60_000])
    lib.build_index(str(tmp_path / "g.fa"), str(tmp_path / "idx"), 16)
    reads = _reads(g0, starts, n, rng)
    want = PortOracle(str(tmp_path / "idx")).search(reads, mode=lib.MODE_SEARCH1, max_results=1 << 16, threads=8)
    assert len(want.hits) > 1000
    with lib.GpuIndex(str(tmp_path / "idx")) as g:
        assert g.full_rows()
        for form in (lib.FORM_BATCHED, lib.FORM_PLAIN):
            got = g.search(reads, mode=lib.MODE_SEARCH1, form=form, max_results=1 << 16)
            assert got.equal(want), f"form {form}"
