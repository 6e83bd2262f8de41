"""Seeds and CALs without the whole suffix arrays."""
from __future__ import annotations

import pytest

from sampled_arrays import sampled_arrays  # noqa: F401
from test_gpu_seeds import (loaded, test_cal_batch_equals_reference, test_seeds_and_cals_match_reference,  # noqa: F401
                            test_short_and_odd_reads, test_single_seed_entry_point)

pytestmark = pytest.mark.gpu
