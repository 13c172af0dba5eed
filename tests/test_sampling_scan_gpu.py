"""The sampling kernel's passes over a row: 16 bytes a load or one element, one block, eight and sixteen, rows that shared memory keeps
and longer ones, blocks without elements, histograms that are emptied on the way (more than 65,532 elements a block).  Sums of masses are integers, so
every form gives the same token."""
import pytest
import torch

import plain_qwen2 as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("R,V", [(2, 4), (6, 1000), (3, 4099), (5, 152064), (128, 155648), (3, 300000), (2, 600004), (131, 2052),
                                 (3, 4096), (3, 4100), (40, 6000), (40, 19456), (40, 19460), (1, 155652), (2, 778240), (2, 778244), (1, 800001)])
@pytest.mark.parametrize("spread", [0.01, 3.0, 12.0])
def test_loads_and_blocks_do_not_change_the_token(R, V, spread):
    from pico_vllm_b200 import ops
    g = torch.Generator().manual_seed(V + R)
    logits = torch.randn(R, V, generator=g) * spread
    temp = torch.tensor([(0.0, 0.7, 1.0, 1.6)[(r + 1) % 4] for r in range(R)])
    top_p = torch.tensor([(1.0, 0.9, 0.999, 0.3, 0.0)[r % 5] for r in range(R)])
    u = torch.rand(R, generator=g)
    wide = torch.empty(R, V + 1, device=DEV)
    wide[:, :V] = logits.to(DEV)
    outs = []
    for x in (logits.to(DEV), wide[:, :V]):
        out = torch.full((R,), -1, dtype=torch.int32, device=DEV)
        ops.sample(x, temp.to(DEV), top_p.to(DEV), u.to(DEV), out)
        outs.append(out.cpu().tolist())
    assert outs[0] == outs[1]
    for r in range(min(R, 5)):
        got = outs[0][r]
        if temp[r] == 0:
            assert got == int(torch.argmax(logits[r]))
            continue
        probs = torch.softmax(logits[r].double() / float(temp[r]), 0)
        if top_p[r] <= 0:
            assert probs[got] == probs.max()        # only the largest is kept
            continue
        if top_p[r] < 1:
            probs = plain.top_p_filter(probs[None], float(top_p[r]))[0]
        cum = torch.cumsum(probs, 0)
        # a weight's float32 exponential is off by 1e-6 of itself, its mass by up to 2^-32 of the largest: over 800,001 of them
        # the kept mass is off by less than 1.9e-4, and so is where the running sum passes the target
        lo, hi, target = float(cum[got] - probs[got]), float(cum[got]), float(u[r]) * float(cum[-1])
        assert lo - 2e-4 <= target <= hi + 2e-4, (r, lo, target, hi)
