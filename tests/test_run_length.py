"""The length of the runs that a prompt of the fading state or the dual form is cut into."""

import pytest

from semantic_aware_adaptive_kv_cache_precision_b200 import ops


@pytest.mark.parametrize("longest,run", [(0, 0), (1, 0), (32, 0), (63, 0), (64, 32), (127, 32),
                                         (128, 64), (129, 64), (100000, 64)])
def test_run_length(longest, run):
    assert ops.run_length(longest) == run


@pytest.mark.parametrize("longest,tokens,sequences,run", [
    (64, 64, 1, 32), (64, 71, 8, 32), (64, 72, 9, 32), (64, 73, 10, 0), (100, 355, 256, 0), (200, 223, 24, 64),
    (200, 240, 41, 0), (2000, 2255, 256, 64), (64, 4096, 64, 32), (63, 63, 1, 0)])
def test_one_walk_where_most_sequences_bring_few_tokens(longest, tokens, sequences, run):
    """A prompt beside many decoded tokens; many prompts are runs."""
    assert ops.run_length(longest, tokens, sequences) == run


def test_the_runs_of_a_step_and_their_memory():
    """A scratch row for every run there can be: one for every `run` tokens of the step and one a sequence."""
    from types import SimpleNamespace

    from semantic_aware_adaptive_kv_cache_precision_b200.ops import scan
    for lengths in ([64], [1] * 255 + [100], [63, 1, 64, 65, 128], [200, 3, 3, 130]):
        step = SimpleNamespace(sequences=len(lengths), max_new=max(lengths))
        runs, scratch, sums = scan._runs(32, step, 6, 2, "cpu", sum(lengths))
        assert runs == -(-max(lengths) // 32)
        assert scratch.shape == (sum(lengths) // 32 + len(lengths), 6) and sums.shape[0] == scratch.shape[0]
        at, row = 0, -1                    # every sequence's rows follow those of the one before
        for b, n in enumerate(lengths):
            first = at // 32 + b
            assert first > row
            row = first + -(-n // 32) - 1
            at += n
        assert row < scratch.shape[0]


@pytest.mark.parametrize("longest,sequences,inner,state,run", [
    (127, 1, 64, 16, 0), (128, 1, 64, 16, 32), (255, 4, 2048, 16, 32), (255, 4, 2369, 16, 0), (128, 37, 256, 16, 32),
    (128, 38, 256, 16, 0), (255, 1, 64, 17, 0), (256, 64, 4096, 16, 64), (256, 1, 64, 128, 64)])
def test_the_selective_scan_s_runs(monkeypatch, longest, sequences, inner, state, run):
    """Shorter runs up to 64 channels an SM, all sequences together; one walk in the 32-bit mode."""
    from types import SimpleNamespace

    import torch

    from semantic_aware_adaptive_kv_cache_precision_b200.parts.selective_scan import SelectiveScanMixer
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    step = SimpleNamespace(max_new=longest, sequences=sequences)
    part = SimpleNamespace(act_dtype=torch.bfloat16, spec=SimpleNamespace(inner=inner, state=state))
    assert SelectiveScanMixer._run(part, step) == run
    part.act_dtype = torch.float32
    assert SelectiveScanMixer._run(part, step) == 0
