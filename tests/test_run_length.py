"""The length of the runs that a prompt of the fading state or the dual form is cut into."""

import pytest

from semantic_aware_adaptive_kv_cache_precision_b200 import ops


@pytest.mark.parametrize("longest,run", [(0, 0), (1, 0), (32, 0), (63, 0), (64, 32), (127, 32),
                                         (128, 64), (129, 64), (100000, 64)])
def test_run_length(longest, run):
    assert ops.run_length(longest) == run
