"""Which steps run their recurrences in blocks."""
from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("counts,heads,blocks", [
    ([112], 2, True), ([111], 64, False), ([600, 1], 1, True),         # one long portion, whatever the heads
    ([32] * 8, 2, False), ([32] * 8, 8, False), ([32] * 8, 16, True),  # several short ones: their scans share the SMs where the heads are many
    ([32] * 16, 8, True), ([27] * 100, 64, False), ([28] * 10, 32, True)])
def test_blocks_where_scans_share_the_sms(counts, heads, blocks):
    import torch
    from kestrel_llm_b200.csrc import ops
    step = SimpleNamespace(max_count=max(counts), num_tokens=sum(counts), captured=False)
    assert ops.recurrence_in_blocks(step, torch.bfloat16, 128, heads) is blocks
    assert not ops.recurrence_in_blocks(step, torch.float32, 128, heads)
    assert not ops.recurrence_in_blocks(step, torch.bfloat16, 129, heads)
    step.captured = True
    assert not ops.recurrence_in_blocks(step, torch.bfloat16, 128, heads)


@pytest.mark.parametrize("counts,by_length", [([500], 0), ([500, 500], 0), ([256] * 8, 0), ([592, 1185], 1), ([1185, 592], 1), ([117, 233, 350], 1), ([16] * 63 + [17], 1),
                                              ([16] * 64 + [17], 0)])
def test_only_unequal_requests_are_scanned_by_length(counts, by_length):
    from kestrel_llm_b200.csrc import ops
    assert ops.library().kestrel_recurrence_blocks_by_length(sum(counts), len(counts), max(counts)) == by_length
