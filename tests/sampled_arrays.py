"""The fixture of the modules that run other modules' tests on the sampled arrays: every index a test opens goes
without the whole suffix arrays and the text, as an index does that finds no room for them."""
from __future__ import annotations

import pytest

from hpgbwt import lib


@pytest.fixture(autouse=True)
def sampled_arrays(monkeypatch):
    class Sampled(lib.GpuIndex):
        def __init__(self, *args, **kwargs):
            super().__init__(*args, **kwargs)
            self.set_full_rows(False)
            assert not self.full_rows()

    monkeypatch.setattr(lib, "GpuIndex", Sampled)
