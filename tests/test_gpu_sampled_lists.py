"""The alignment lists without the whole suffix arrays."""
from __future__ import annotations

import pytest

from sampled_arrays import sampled_arrays  # noqa: F401
from test_gpu_api import (loaded, test_array_list_form, test_batch_forms_equal_per_read,  # noqa: F401
                          test_entry_points_match_reference)

pytestmark = pytest.mark.gpu
