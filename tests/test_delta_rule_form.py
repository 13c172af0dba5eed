"""Which form the recurrence with a decay per head takes: by the blocks that are at work, counted over heads, columns and segments."""
import pytest
import torch

from pico_vllm_b200 import ops


@pytest.mark.parametrize("heads,lens,dv,take", [
    (12, [512], 128, True), (37, [512], 128, True), (38, [512], 128, False), (48, [2048], 128, False), (48, [2048], 96, True),     # one segment: 296 blocks
    (8, [512] * 4, 128, False), (8, [528] * 4, 128, True), (12, [600] * 4, 128, False), (12, [683] * 3, 128, True), (13, [683] * 3, 128, False),
    (12, [1025, 682, 341], 128, True), (16, [1025, 682, 341], 128, True), (24, [1025, 682, 341], 128, False),
    (12, [1024] + [96] * 16, 128, True), (12, [1024] + [150] * 16, 128, False),
    (12, [992] + [1] * 60, 128, True), (12, [991] + [1] * 60, 128, False), (16, [1024] + [1] * 60, 128, False), (16, [1152] + [1] * 60, 128, True),
    (24, [1024] + [1] * 60, 128, False),
])
def test_chunks_where_the_longest_segment_sets_the_time(heads, lens, dv, take):
    T, S = sum(lens), len(lens)
    v, state = torch.empty(T, heads * dv), torch.empty(1, heads, dv, 128)
    assert ops.delta_chunks_take(v, state, 128, dv, max(lens), S) == take
