"""Parts of the key range in steps that hold portions of prompts beside single tokens."""
import pytest
import torch

from pico_vllm_b200 import ops
from pico_vllm_b200.config import EngineConfig
from pico_vllm_b200.parts import GQAAttention, Rotary
from pico_vllm_b200.parts import attention
from pico_vllm_b200.parts.base import StepShape


def _plan(q_lens, starts, dtype="bfloat16", heads=28, kv=4, sms=148, pad=0):
    part = GQAAttention(512, heads, kv, 128, position=Rotary(128, 1e6))
    T = sum(q_lens) + pad
    return part.plan(StepShape(num_tokens=T, num_segments=len(q_lens) + pad, q_lens=q_lens, starts=starts,
                               max_kv=max(n + s for n, s in zip(q_lens, starts)), decode_only=max(q_lens) == 1, num_sms=sms,
                               engine=EngineConfig(dtype=dtype)))


def test_only_single_tokens_are_counted_beside_portions():
    alone = _plan([1] * 8, [3000] * 8)
    assert alone.splits == 8
    assert _plan([1] * 8 + [500], [3000] * 8 + [0]).splits == alone.splits
    assert _plan([500, 1], [0, 3000]).splits == 16                   # few blocks: as a batch of one
    assert _plan([500, 1], [4000, 100]).splits == 1                  # a long portion does not split a short single token
    assert _plan([500], [3000]).splits == 1
    assert _plan([500], [3000], pad=1).splits == 1                   # a padding row holds no keys


def test_short_contexts_beside_portions_stay_whole():
    assert _plan([419, 406] + [1] * 27, [0] + [504] * 28, heads=16, kv=2).splits == 1
    assert _plan([500] + [1] * 8, [0] + [1022] * 8).splits == 1
    assert _plan([500] + [1] * 8, [0] + [1023] * 8).splits == _plan([1] * 8, [1023] * 8).splits == 8
    assert _plan([6] + [1] * 8, [0] + [600] * 8).splits == _plan([1] * 14, [600] * 14).splits == 4     # few tokens: as if all were single


def test_scratch_for_every_token_bounds_the_parts():
    plan = _plan([1] * 8 + [2040], [3000] * 8 + [0])
    assert plan.splits == 4 and plan.scratch_floats == 2048 * 28 * 4 * 130 <= attention.MAX_MIXED_SCRATCH < 2048 * 28 * 8 * 130
    plan = _plan([1] * 8 + [5000], [3000] * 8 + [0])
    assert plan.splits == 1 and plan.scratch_floats == 0 and 5008 * 28 * 2 * 130 > attention.MAX_MIXED_SCRATCH


def test_the_32_bit_path_still_counts_every_token():
    assert _plan([1] * 8 + [500], [3000] * 8 + [0], dtype="float32").splits == 1


@pytest.mark.parametrize("H,G,hd,q_lens,starts,want", [
    (12, 2, 128, [333] + [1] * 7, [0] + [777] * 7, (4, 0)), (12, 2, 128, [333], [0], (0, 0)), (12, 2, 128, [333], [306], (0, 0)),
    (12, 2, 128, [333], [307], (4, 0)), (12, 2, 128, [199] + [1] * 8, [0] + [700] * 8, (4, 128)), (12, 2, 128, [200] + [1] * 8, [0] + [700] * 8, (4, 128)),
    (12, 2, 128, [1479], [0], (4, 0)), (12, 2, 128, [1480], [0], (0, 0)), (8, 8, 64, [333] + [1] * 7, [0] + [777] * 7, (4, 128)),
    (8, 8, 64, [40], [1000], (4, 128)), (4, 1, 256, [500], [500], (0, 0)), (4, 1, 256, [600], [500], (4, 0)), (12, 2, 128, [2, 1], [3000, 3000], (0, 0)),
    (2000, 500, 128, [40], [1000], (0, 0)),
    # many single tokens already fill the device; a few do not
    (12, 2, 128, [2] + [1] * 200, [700] * 201, (0, 0)), (12, 2, 128, [2] + [1] * 64, [850] * 65, (0, 0)), (32, 8, 128, [63] + [1] * 64, [1700] * 65, (0, 0)),
    (12, 2, 128, [17] + [1] * 64, [0] + [100] * 63 + [1000], (4, 128)),
    # portions that fit at once, of a quarter of a round more
    (28, 4, 128, [110, 1], [1250, 1000], (0, 0)), (28, 4, 128, [140, 1], [1250, 1000], (4, 0)),
    # of both: by the load, and by the rows of a block of 8 that a head's queries leave empty
    (12, 2, 128, [150, 137] + [1] * 8, [0, 185, 401, 282, 242, 714, 197, 294, 426, 201], (4, 0)),
    (16, 2, 128, [150, 137] + [1] * 8, [0, 185, 401, 282, 242, 714, 197, 294, 426, 201], (4, 128)),
    # short contexts
    (12, 2, 128, [17] * 3 + [1], [0] * 3 + [382], (0, 0)), (12, 2, 128, [60], [500], (0, 0)), (12, 2, 128, [40] + [1] * 8, [0] + [510] * 8, (0, 0)),
    (12, 2, 128, [40] + [1] * 8, [0] + [511] * 8, (4, 128))])
def test_parts_of_float32_steps_with_portions(H, G, hd, q_lens, starts, want):
    part = GQAAttention(H * hd, H, G, hd, position=Rotary(hd, 1e6))
    shape = StepShape(num_tokens=sum(q_lens), num_segments=len(q_lens), q_lens=q_lens, starts=starts, max_kv=max(a + b for a, b in zip(q_lens, starts)),
                      decode_only=False, num_sms=148, engine=EngineConfig(dtype="float32"))
    plan = part.plan(shape)
    assert (plan.run_parts, plan.part_keys) == want and plan.key == (plan.splits, 0) + want
    assert plan.scratch_floats == ops.attention_scratch_floats(shape.num_tokens, H, hd, max(plan.splits, want[0]))


@pytest.mark.parametrize("graph", [False, True])
def test_a_float32_step_without_room_for_its_parts_goes_without_them(graph, monkeypatch):
    """The device's pages leave no room: the allocator's own error leads to the plan that needs no scratch, and a full portion is recorded with it."""
    import helpers
    from pico_vllm_b200.engine import StepItem
    import fake_ops
    fake_ops.install(monkeypatch)
    runner, _ = helpers.make_runner_from_tensors("a", "float32", "cpu", 2048)
    monkeypatch.setattr(GQAAttention, "_run_parts", lambda self, shape, splits: (4, 128) if shape.spare else (0, 0))
    slot = runner.cache.acquire("x")
    item, plans = StepItem(slot, helpers.random_ids(700, 256, 5), (699,)), []
    if graph:
        monkeypatch.setattr(runner, "on_gpu", True)
        monkeypatch.setattr(runner.cfg, "use_cuda_graph", True)
        runner._graph_prefill_tokens = 700
        monkeypatch.setattr(runner, "_run_and_record", lambda key, batch, entry: (runner._graphs.setdefault(key, entry), plans.append((batch.plans, batch.scratch))))
    else:
        forward = runner.model.forward
        monkeypatch.setattr(runner.model, "forward", lambda batch, views: (plans.append((batch.plans, batch.scratch)), forward(batch, views))[1])

    def full(need):
        if need > 0:
            raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(runner, "_new_scratch", full)
    runner.step([item])
    (plan,), scratch = plans[0][0].values(), plans[0][1]
    assert plan.run_parts == 0 and plan.scratch_floats == 0 and scratch is None
