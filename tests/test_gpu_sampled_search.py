"""The searches, the block search and the server without the whole suffix arrays: the warp-cooperative form with its
settings, long reads and overflowing stacks, LF locate with its limit, plans that grow, served batches."""
from __future__ import annotations

import pytest

from sampled_arrays import sampled_arrays  # noqa: F401
from test_gpu_block import (golden, test_array_list_2_equals_per_read,  # noqa: F401
                            test_block_search_matches_reference_fixtures,
                            test_block_search_repetitive_reads_and_locate_limit)
from test_gpu_graph import (copies_case, test_device_bases_at_any_address, test_graph_batches_of_every_size,  # noqa: F401
                            test_graph_device_entry, test_graph_pools_grow, test_graph_rejects_bad_offsets,
                            test_graph_replay_launches_counted, test_pipelined_host_batches)
from test_gpu_parity import (test_batched_golden, test_block_load_modes_agree, test_edge_reads,  # noqa: F401
                             test_gpu_matches_oracle, test_large_intervals_match_oracle,
                             test_locate_limit_matches_oracle, test_start_table_lengths_agree,
                             test_truncation_matches_oracle, test_wave_form_agrees, test_wave_long_reads,
                             test_wave_overflowing_stacks, test_wave_start_table_and_truncation)
from test_gpu_serve import (test_alone_equals_in_mix, test_batches_share_requests_and_budget_splits_them,  # noqa: F401
                            test_serving_locate_limit, test_serving_pools_grow)

pytestmark = pytest.mark.gpu
