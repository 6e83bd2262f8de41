"""The search with the text, suffix array and inverse on the device against the oracle and against the sampled
arrays (the general path): read lengths around the start table, the packed words and the branching windows, reads
at both ends of the text and across chromosomes, repeats wider than a warp's stack, every complement pairing."""
from __future__ import annotations

import numpy as np
import pytest

from hpgbwt import lib, synth
from oracle.pyoracle import PortOracle

pytestmark = pytest.mark.gpu

_A = np.frombuffer(b"ACGT", dtype=np.uint8)


def _edge_reads(g: np.ndarray, seed: int) -> synth.ReadSet:
    """Reads of every length 3..72 and some longer ones: at the text's two ends and inside, either strand, exact and
    with each kind of edit at the first, last, middle and random positions."""
    rng = np.random.default_rng(seed)
    out = []
    for L in list(range(3, 73)) + [95, 96, 97, 127, 128, 129, 160, 161, 193, 300]:
        for p in (0, 1, len(g) - L, len(g) - L - 1, int(rng.integers(0, len(g) - L))):
            f = g[p:p + L]
            at = [0, 1, L // 2 - 1, L // 2, L // 2 + 1, L - 2, L - 1, int(rng.integers(0, L))][int(rng.integers(0, 8))]
            at = min(max(at, 0), L - 1)
            sub = f.copy()
            sub[at] = (sub[at] + rng.integers(1, 4)) % 4
            ins = np.insert(f, at, rng.integers(0, 4)).astype(np.uint8)
            dele = np.delete(f, at)
            for r in (f, sub, ins, dele):
                if len(r) >= 3:
                    out.append(_A[r if rng.random() < 0.5 else synth.revcomp_codes(r)].tobytes())
    return synth.from_strings(out)


def _check(g: lib.GpuIndex, reads, want, max_results):
    for rows in (True, False):
        assert g.set_full_rows(rows) == rows
        for graph in (True, False):
            g.set_graph(graph)
            got = g.search(reads, mode=lib.MODE_SEARCH1, form=lib.FORM_BATCHED, max_results=max_results)
            assert got.equal(want), f"full rows {rows}, graph {graph}"
        got = g.search(reads, mode=lib.MODE_SEARCH1, form=lib.FORM_PLAIN, max_results=max_results)
        assert got.equal(want), f"plain form, full rows {rows}"


@pytest.mark.parametrize("kind,n,chroms", [("iid", 700, 1), ("iid", 30_011, 2), ("repeats", 200_000, 3),
                                           ("human_like", 60_000, 2)])
def test_edges_match_oracle(case_factory, kind, n, chroms):
    c = case_factory(kind, n, 31, chroms)
    reads = _edge_reads(c.genome, 5)
    want = PortOracle(c.index).search(reads, mode=lib.MODE_SEARCH1, max_results=1 << 16, threads=8)
    with lib.GpuIndex(c.index) as g:
        assert g.full_rows()
        _check(g, reads, want, 1 << 16)


@pytest.mark.parametrize("symbols", [0, 8, 12])
@pytest.mark.parametrize("max_results", [2, 1 << 16])
def test_start_tables_and_repeats(case_factory, symbols, max_results):
    c = case_factory("human_like", 200_000, 3, 5)
    reads = synth.reads(c.genome, 3000, 19, length=(20, 140), edits="mix_30_50_20")
    want = PortOracle(c.index).search(reads, mode=lib.MODE_SEARCH1, max_results=max_results, threads=8)
    with lib.GpuIndex(c.index) as g:
        g.set_start_table(symbols)
        _check(g, reads, want, max_results)


@pytest.mark.parametrize("bases", ["ACGT", "ATCG", "ACTG"])
def test_complement_pairings(tmp_path, bases):
    gen = synth.genome("repeats", 50_000, 8)
    synth.write_fasta(str(tmp_path / "g.fa"), gen, [20_000, 30_000])
    lib.build_index(str(tmp_path / "g.fa"), str(tmp_path / "idx"), 16, bases=bases)
    reads = synth.reads(gen, 1500, 4, length=(30, 110), edits="mix_30_50_20")
    want = PortOracle(str(tmp_path / "idx")).search(reads, mode=lib.MODE_SEARCH1, max_results=1 << 16, threads=8)
    assert len(want.hits) > 1000
    with lib.GpuIndex(str(tmp_path / "idx")) as g:
        _check(g, reads, want, 1 << 16)


@pytest.mark.parametrize("ratio", [1, 10, 32])
def test_sampling_ratios(tmp_path, ratio):
    """The derivation walks from the index's own samples, at any ratio."""
    gen = synth.genome("iid", 20_000, 12)
    synth.write_fasta(str(tmp_path / "g.fa"), gen)
    lib.build_index(str(tmp_path / "g.fa"), str(tmp_path / "idx"), ratio)
    reads = synth.reads(gen, 800, 2, length=(20, 90), edits="mix_30_50_20")
    want = PortOracle(str(tmp_path / "idx")).search(reads, mode=lib.MODE_SEARCH1, max_results=1 << 16, threads=8)
    with lib.GpuIndex(str(tmp_path / "idx")) as g:
        assert g.full_rows()
        _check(g, reads, want, 1 << 16)


@pytest.mark.parametrize("kind,n", [("iid", 700), ("human_like", 60_000)])
def test_exact_search_edges(case_factory, kind, n):
    """The exact search from its graph, from device or host bases, against the oracle and the plain form."""
    c = case_factory(kind, n, 31, 2)
    reads = _edge_reads(c.genome, 6)
    want = PortOracle(c.index).search(reads, mode=lib.MODE_EXACT, max_results=1, threads=8)
    with lib.GpuIndex(c.index) as g:
        for rows in (True, False):
            g.set_full_rows(rows)
            for max_results in (1, 0):  # an exact list holds one hit whatever the capacity
                for form in (lib.FORM_BATCHED, lib.FORM_PLAIN):
                    got = g.search(reads, mode=lib.MODE_EXACT, form=form, max_results=max_results)
                    assert got.equal(want), f"full rows {rows}, form {form}, capacity {max_results}"
        g.set_locate_limit(1)
        a = g.search(reads, mode=lib.MODE_EXACT, form=lib.FORM_BATCHED)
        assert a.equal(g.search(reads, mode=lib.MODE_EXACT, form=lib.FORM_PLAIN))
        bad = synth.ReadSet(reads.seq, reads.offsets.copy(), reads.truth_pos, reads.truth_strand, reads.edit)
        bad.offsets[5] = bad.offsets[7] + np.uint64(1)
        with pytest.raises(RuntimeError, match="non-decreasing"):
            g.search(bad, mode=lib.MODE_EXACT, form=lib.FORM_BATCHED)
