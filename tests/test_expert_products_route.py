"""Which routed feed-forwards run on the tcgen05 tensor cores."""
import pytest
import torch

from pico_vllm_b200 import ops


def _takes(E, pairs, D=64, ff=64, gated=True, dtype=torch.bfloat16):
    h, up, down = torch.empty(pairs, D, dtype=dtype), torch.empty(E, (2 if gated else 1) * ff, D, dtype=dtype), torch.empty(E, D, ff, dtype=dtype)
    return ops.moe_tc_takes(h, up, down, pairs)


@pytest.mark.parametrize("E,pairs,take", [(16, 256, False), (16, 257, True), (512, 8193, True), (513, 8209, True), (1024, 16385, True), (1025, 16401, False)])
def test_experts(E, pairs, take):
    assert _takes(E, pairs) == take
    assert not _takes(E, pairs, dtype=torch.float32)
