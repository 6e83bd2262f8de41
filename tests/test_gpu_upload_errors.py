"""A call that fails for want of device memory after its reads were queued for upload returns with nothing in flight:
the caller may free or rewrite its page-locked arrays at once."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from hpgbwt import lib, synth

pytestmark = pytest.mark.gpu


def test_no_copy_outlives_a_failed_block_search(case_factory):
    torch = pytest.importorskip("torch")
    c = case_factory("iid", 200_000, 9, 2)
    n, L = 10_000_000, 100
    offs = torch.arange(0, (n + 1) * L, L, dtype=torch.int64).pin_memory()
    seq = torch.full((n * L,), 65, dtype=torch.uint8).pin_memory()
    small = synth.reads(c.genome, 500, 3, length=80, edits="mix_30_50_20")
    with lib.GpuIndex(c.index) as g:
        want = g.block_search(small)
        stream = torch.cuda.ExternalStream(g.stream())
        torch.cuda.empty_cache()
        # room for the reads (2.4 GB with their codes), not for the search's 8 GB
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (4 << 30), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        rs = lib.ResultSetC()
        rc = g.lib.bwt_gpu_block_search(g.handle, seq.data_ptr(), offs.data_ptr(), n, 16, ctypes.byref(rs), None, None)
        idle = stream.query()
        msg = g.lib.bwt_gpu_last_error().decode()
        stream.synchronize()
        del fill
        torch.cuda.empty_cache()
        assert rc != 0 and "block search" in msg
        assert idle, "the failed call left copies from the caller's arrays in flight"
        assert g.block_search(small).equal(want)
