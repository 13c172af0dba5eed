"""How many parts a single token's keys are cut into: by the contexts' lengths and by how even they are."""
from dataclasses import replace

import pytest

from pico_vllm_b200.config import EngineConfig
from pico_vllm_b200.parts import GQAAttention, Rotary
from pico_vllm_b200.parts.attention import QKNormAttention, decode_splits
from pico_vllm_b200.parts.biased_attention import DistanceBiasAttention
from pico_vllm_b200.parts.base import StepShape


def _splits(contexts, kv_heads, dtype="bfloat16", window=None, cluster=True):
    n = len(contexts)
    shape = StepShape(num_tokens=n, num_segments=n, q_lens=[1] * n, starts=[c - 1 for c in contexts], max_kv=max(contexts),
                      decode_only=True, num_sms=148, engine=EngineConfig(dtype=dtype))
    return decode_splits(shape, kv_heads, window, cluster)


@pytest.mark.parametrize("contexts,kv_heads,parts,before", [
    ([200], 2, 1, 1), ([255], 2, 1, 1), ([256], 2, 4, 2), ([512], 2, 8, 4), ([1500], 2, 8, 8), ([2048], 2, 16, 16),
    ([500] * 32, 4, 1, 2), ([511] * 32, 4, 1, 2), ([512] * 32, 4, 2, 2), ([1024] * 32, 4, 2, 2),                # two parts at most
    ([512] * 18, 1, 8, 4), ([512] * 19, 1, 4, 4), ([512] * 32, 1, 4, 4), ([1024] * 32, 1, 8, 8),                # eight: a block per SM
    ([300] * 32, 2, 4, 2), ([300] * 64, 1, 4, 2), ([300] * 65, 1, 1, 2), ([504] * 37, 2, 1, 2), ([511] * 37, 2, 1, 2), ([512] * 37, 2, 4, 4),
    ([8000] * 40, 4, 1, 1), ([8000] + [3000] * 39, 4, 4, 1), ([4095] + [1000] * 39, 4, 1, 1), ([4096] + [1000] * 39, 4, 4, 1),
])
def test_parts(contexts, kv_heads, parts, before):
    assert _splits(contexts, kv_heads) == parts
    assert _splits(contexts, kv_heads, "float32") == before
    assert _splits(contexts, kv_heads, cluster=False) == before         # kernels whose parts a second launch adds up


def test_portions_that_are_counted_keep_ragged_batches_whole():
    shape = StepShape(num_tokens=2040, num_segments=41, q_lens=[2000] + [1] * 40, starts=[0, 7999] + [2999] * 39, max_kv=8000,
                      decode_only=False, num_sms=148, engine=EngineConfig(dtype="bfloat16"))
    assert decode_splits(shape, 4) == 1
    assert decode_splits(replace(shape, num_tokens=40), 4) == 4


def test_a_window_bounds_the_keys():
    assert _splits([8000] + [3000] * 39, 4, window=4000) == 1
    assert _splits([8000] + [100] * 39, 4, window=5000) == 4
    assert _splits([8000], 2, window=300) == 4


@pytest.mark.parametrize("part,clustered", [
    (lambda: GQAAttention(512, 12, 2, 128, position=Rotary(128, 1e6)), True), (lambda: GQAAttention(512, 12, 2, 96, position=Rotary(96, 1e6)), False),
    (lambda: GQAAttention(512, 34, 2, 128, position=Rotary(128, 1e6)), False),                       # 17 query heads a kv head
    (lambda: QKNormAttention(512, 12, 2, 64, Rotary(64, 1e6), 1e-6), True), (lambda: QKNormAttention(512, 12, 2, 80, Rotary(80, 1e6), 1e-6), False),
    (lambda: DistanceBiasAttention(512, 12, 2, 64, 128, 1e-6), True), (lambda: DistanceBiasAttention(512, 12, 2, 64, 128, 1e-6, chunk=4096), False),
])
def test_short_parts_only_where_a_cluster_adds_them_up(part, clustered):
    shape = StepShape(num_tokens=4, num_segments=4, q_lens=[1] * 4, starts=[511] * 4, max_kv=512, decode_only=True, num_sms=148,
                      engine=EngineConfig(dtype="bfloat16", page_size=16))
    assert part().plan(shape).splits == (8 if clustered else 4)
    assert part().plan(replace(shape, engine=EngineConfig(dtype="bfloat16", page_size=24))).splits == 4


@pytest.mark.parametrize("batch,kv_heads,parts", [(64, 4, 4), (65, 4, 1), (128, 2, 4), (130, 2, 1), (512, 8, 1)])
def test_ragged_batches_of_many_requests_stay_whole(batch, kv_heads, parts):
    assert _splits([8000] + [300] * (batch - 1), kv_heads) == parts
