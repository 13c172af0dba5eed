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


def test_narrow_experts_need_many_rows():
    assert not _takes(4, 1023, 1024, 48) and _takes(4, 1024, 1024, 48)
    assert not _takes(4, 1024, 48, 336) and _takes(4, 1024, 48, 344)


@pytest.mark.parametrize("D,ff,take", [(16, 1024, True), (48, 24, False), (1024, 48, True), (2048, 8, False), (8, 2048, False), (1024, 20, False), (36, 1024, False)])
def test_widths(D, ff, take):
    assert _takes(4, 1024, D, ff) == take and _takes(4, 1024, D, ff, gated=False) == take
