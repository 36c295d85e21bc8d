"""Which form a kernel with several takes at which sizes (no GPU needed; on 148 SMs): what was measured to be
the faster one. That the forms agree is tested in `test_tile_forms_gpu.py`."""

import pytest

from semantic_aware_adaptive_kv_cache_precision_b200.ops._lib import plain_function


@pytest.mark.parametrize("tokens,outputs,tiles", [(64, 36, 0), (64, 128, 0), (400, 16, 0), (3200, 2, 0), (100000, 2, 0),
                                                  (800, 16, 1), (400, 36, 1), (100, 128, 1), (3200, 4, 1),
                                                  (2 ** 20, 4096, 1)])
def test_router_logits_in_tiles_only_where_there_are_many(tokens, outputs, tiles):
    assert plain_function("sakv_moe_logits_in_tiles")(tokens, outputs) == tiles


@pytest.mark.parametrize("tokens,width,by_tokens", [(8, 1024, 0), (64, 1024, 0), (4096, 64, 0), (4096, 128, 0),
                                                    (1024, 256, 1), (256, 1024, 1), (4096, 2048, 1)])
def test_a_token_a_block_sums_the_experts_rows_only_in_long_steps(tokens, width, by_tokens):
    assert plain_function("sakv_moe_combine_by_tokens")(tokens, width) == by_tokens


@pytest.mark.parametrize("tokens,channels,taps,runs", [(9, 4096, 4, 0), (128, 1024, 4, 0), (64, 2304, 4, 0),
                                                       (64, 4096, 4, 1), (256, 1024, 4, 1), (3400, 4096, 4, 1),
                                                       (3400, 4096, 3, 0)])
def test_eight_tokens_a_thread_in_the_convolution_only_in_long_steps(tokens, channels, taps, runs):
    assert plain_function("sakv_conv_by_runs")(tokens, channels, taps) == runs
