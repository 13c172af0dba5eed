"""The delta rule with a decay per head in chunks of 32 tokens against the recurrence token by token in float64: the edges of
chunks, single tokens and padding beside them, key sizes that are padded, column tiles that are not full, decays of nought and one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _segments(lens, pad_at=None):
    cu, pos = [0], []
    for s, n in enumerate(lens):
        cu.append(cu[-1] + n)
        pos += [-1] * n if s == pad_at else list(range(5 * s, 5 * s + n))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32)
    return i32(cu), i32(pos), i32(list(range(len(lens) - 1, -1, -1)))


def _oracle(q, k, v, a, beta, state, slots, cu, pos):
    T, H, dv = v.shape
    G = q.shape[1]
    out, state = torch.zeros(T, H, dv, dtype=torch.float64), state.double().clone()
    q, k = (x.double().repeat_interleave(H // G, 1) for x in (q, k))
    for s in range(slots.shape[0]):
        a0, a1 = int(cu[s]), int(cu[s + 1])
        if a1 <= a0 or int(pos[a0]) < 0:
            continue
        S = state[int(slots[s])]                                  # [H, dv, d]
        for t in range(a0, a1):
            S = S * a[t].double()[:, None, None]
            u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hvd,hd->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None, :]
            out[t] = torch.einsum("hvd,hd->hv", S, q[t])
        state[int(slots[s])] = S
    return out, state


@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 128, 128), (3, 3, 68, 20), (10, 2, 100, 36), (1, 1, 128, 4)])
@pytest.mark.parametrize("lens,pad_at", [([64], None), ([1, 31, 32, 33, 70, 1], None), ([97, 5, 2, 64], 1), ([0, 128, 0, 65], None)])
@pytest.mark.parametrize("decays,off", [("middling", 0), ("nought and one", 0), ("middling", 1)])
def test_chunks(H, G, d, dv, lens, pad_at, decays, off, monkeypatch):
    _check(H, G, d, dv, lens, pad_at, decays, off, monkeypatch)


@pytest.mark.parametrize("H,G,d,dv,lens,blocks", [
    (28, 28, 68, 20, [320], 294), (29, 29, 68, 20, [320], 304), (58, 29, 128, 128, [320], 304), (52, 26, 100, 128, [31, 65, 224], 299),
    (42, 42, 100, 36, [320], 441), (84, 42, 128, 128, [320], 441), (43, 43, 128, 4, [320], 451), (56, 56, 68, 20, [320], 588),
    (57, 57, 100, 36, [320], 598), (168, 84, 72, 128, [320], 882), (85, 85, 68, 8, [320], 892)])
def test_three_blocks_a_multiprocessor_prepare(H, G, d, dv, lens, blocks, monkeypatch):
    """Chunks times key heads at both ends of the ranges in which three blocks a multiprocessor save a round (297 to 444 and 593 to 888 of
    148 multiprocessors) and outside them, values narrower and wider than the queries whose place they take."""
    assert (2 * (sum(lens) // 32) + min(len(lens), sum(lens) // 64)) * G // 2 == blocks
    _check(H, G, d, dv, lens, None, "middling", 0, monkeypatch)


def _check(H, G, d, dv, lens, pad_at, decays, off, monkeypatch):
    from pico_vllm_b200 import ops
    monkeypatch.setattr(ops, "delta_chunks_take", lambda *a: True)
    g = torch.Generator().manual_seed(d + dv + len(lens))
    cu, pos, slots = _segments(lens, pad_at)
    T, S = int(cu[-1]), len(lens)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, d, generator=g), dim=-1) for _ in range(2))
    q = q * d ** -0.5
    k[1::3] = k[0::3][:k[1::3].shape[0]]                          # keys that repeat: what is held under them is taken off
    v = torch.randn(T, H, dv, generator=g)
    a = torch.rand(T, H, generator=g) * 0.2 + 0.8 if decays == "middling" else (torch.rand(T, H, generator=g) > 0.1).float()
    beta = torch.rand(T, H, generator=g)
    state = torch.randn(S + 1, H, dv, d, generator=g) * 0.3
    dots = torch.full((T, G, 8), float("nan"))                    # with the same row's key and the three before, for short segments
    dots[:, :, 0] = (q * k).sum(-1)
    for j in range(3):
        dots[j + 1:, :, 1 + j] = (q[j + 1:] * k[:T - j - 1]).sum(-1)
        dots[j + 1:, :, 4 + j] = (k[j + 1:] * k[:T - j - 1]).sum(-1)
    prep = torch.cat([q.reshape(T, -1), k.reshape(T, -1), torch.stack([a, beta, a * float("nan"), beta], -1).reshape(T, -1),
                      dots.reshape(T, -1)], 1).contiguous()
    want_o, want_s = _oracle(q, k, v, a, beta, state, slots, cu, pos)
    wide = torch.cat([torch.zeros(T, 4), v.reshape(T, -1)], 1).to(DEV)
    got_s, p = state.to(DEV), prep.to(DEV)
    if off:                                                       # rows off 16 bytes: nothing in chunks
        p = torch.cat([torch.zeros(off, device=DEV), p.flatten()])[off:].view(p.shape)
    got_o = ops.gated_delta_rule(p, wide[:, 4:], got_s, slots.to(DEV), cu.to(DEV), pos.to(DEV), H, G, d, dv, per_head=True,
                                 max_q_len=max(lens))
    live = pos >= 0
    # float32 sums of up to d + 32 products of order one, through a forward substitution of 32 rows
    for got, want in ((got_o.cpu().view(T, H, dv)[live], want_o[live]), (got_s.cpu(), want_s)):
        worst = float((got.double() - want).abs().max())
        assert worst <= 2e-5 * max(1.0, float(want.abs().max())), worst


@pytest.mark.parametrize("lens,d,take", [([511], 128, False), ([512], 128, True), ([2048], 64, False), ([2048], 130, False), ([512, 500], 68, False),
                                         ([520, 500], 68, True), ([591] + [1] * 60, 128, False), ([592] + [1] * 60, 128, True), ([300000], 128, False)])
def test_which_steps_go_in_chunks(lens, d, take):
    from pico_vllm_b200 import ops
    T, S = sum(lens), len(lens)
    v, state = torch.empty(T, 2 * 128, device=DEV), torch.empty(S, 2, 128, d, device=DEV)
    assert ops.delta_chunks_take(v, state, d, 128, max(lens), S) == take
    assert not ops.delta_chunks_take(v[:, 1:], state, d, 128, max(lens), S)


@pytest.mark.parametrize("lens,launches", [([512], 3), ([600, 64], 3), ([600, 63], 4)])
def test_no_launch_for_short_segments_that_are_not_there(lens, launches):
    from pico_vllm_b200 import ops
    H, d, T, S = 2, 68, sum(lens), len(lens)
    cu, pos, slots = (t.to(DEV) for t in _segments(lens))
    prep, v, state = torch.zeros(T, 2 * H * d + 12 * H, device=DEV), torch.ones(T, H * 4, device=DEV), torch.zeros(S, H, 4, d, device=DEV)
    before = ops.launches
    out = ops.gated_delta_rule(prep, v, state, slots, cu, pos, H, H, d, 4, per_head=True, max_q_len=max(lens), min_q_len=min(lens))
    assert ops.launches - before == launches and not out.any()


@pytest.mark.parametrize("lens", [[520], [600, 70, 3]])
def test_without_room_for_its_scratch_a_step_goes_without_chunks(lens, monkeypatch):
    """The same outputs and memory, from the allocator's own error on; one segment's rows come without the dot products of neighbours."""
    from pico_vllm_b200 import ops
    H, d, dv, T, S = 2, 68, 8, sum(lens), len(lens)
    g = torch.Generator().manual_seed(T)
    cu, pos, slots = (t.to(DEV) for t in _segments(lens))
    xc, proj = torch.randn(T, H * (2 * d + dv), generator=g).to(DEV), torch.randn(T, 2 * H, generator=g).to(DEV)
    bias, state = torch.zeros(H, device=DEV), torch.randn(S, H, dv, d, generator=g).to(DEV)
    prep = ops.delta_prepare(xc, 0, H * d, proj, 0, proj[:, H:], bias, bias, H, H, d, per_head=True, max_q_len=1 if S == 1 else max(lens))
    real, asked, got = torch.empty, [], []

    def empty(*size, **how):
        if size and isinstance(size[0], int):
            asked.append(size[0])
            raise torch.OutOfMemoryError("no room")
        return real(*size, **how)
    for full in (False, True):
        if full:
            monkeypatch.setattr(torch, "empty", empty)
        after = state.clone()
        out = ops.gated_delta_rule(prep, xc[:, 2 * H * d:], after, slots, cu, pos, H, H, d, dv, per_head=True, max_q_len=max(lens))
        got.append((out, after))
    assert len(asked) == 1
    for a, b in zip(*got):
        assert torch.allclose(a, b, atol=2e-5 * max(1.0, float(a.abs().max())), rtol=0)


@pytest.mark.parametrize("bad", [0, 5, 31, 32, 45, 69])
@pytest.mark.parametrize("where", ["v", "k", "q", "beta", "decay"])
def test_what_is_no_number_does_not_reach_the_tokens_before_it(where, bad, monkeypatch):
    """A value, key, query, write strength or decay of one head that is no number: the outputs of the tokens before it and of the
    heads that have no part in it stay what they are, bit for bit (a query's also of the tokens after it)."""
    from pico_vllm_b200 import ops
    monkeypatch.setattr(ops, "delta_chunks_take", lambda *a: True)
    H, G, d, dv, T = 4, 2, 128, 36, 70
    g = torch.Generator().manual_seed(bad)
    cu, pos, slots = _segments([T])
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, d, generator=g), dim=-1) for _ in range(2))
    v = torch.randn(T, H, dv, generator=g)
    ab = torch.rand(T, H, 4, generator=g)
    state = torch.randn(1, H, dv, d, generator=g) * 0.3
    outs = []
    for spoil in (False, True):
        if spoil:
            {"v": v[bad, 1], "k": k[bad, 0], "q": q[bad, 0], "beta": ab[bad, 1, 1:2], "decay": ab[bad, 1, :1]}[where].fill_(float("inf") if where in "vq" else float("nan"))
        prep = torch.cat([q.reshape(T, -1), k.reshape(T, -1), ab.reshape(T, -1), torch.zeros(T, 8 * G)], 1).to(DEV)
        outs.append(ops.gated_delta_rule(prep, v.reshape(T, -1).to(DEV), state.to(DEV), slots.to(DEV), cu.to(DEV), pos.to(DEV), H, G, d, dv,
                                         per_head=True, max_q_len=T).cpu().view(T, H, dv))
    clean, got = outs
    reached = [0, 1] if where in "kq" else [1]
    others = [h for h in range(H) if h not in reached]
    assert clean.isfinite().all() and torch.equal(got[:, others], clean[:, others])
    assert torch.equal(got[:bad], clean[:bad])
    assert not got[bad][reached].isfinite().any()
    if where == "q":
        assert torch.equal(got[bad + 1:], clean[bad + 1:])


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), 3e38])
@pytest.mark.parametrize("d,row,col", [(128, 0, 0), (128, 127, 15), (68, 66, 9)])
def test_an_infinity_in_the_memory_stays_in_its_column(value, d, row, col, monkeypatch):
    """A column of the memory that holds an infinity (or a number whose parts for the tensor cores are none): the column's outputs are
    what float32 arithmetic makes of it, and the other columns stay what they are, bit for bit."""
    from pico_vllm_b200 import ops
    monkeypatch.setattr(ops, "delta_chunks_take", lambda *a: True)
    T, dv = 70, 20
    g = torch.Generator().manual_seed(d + row)
    cu, pos, slots = (t.to(DEV) for t in _segments([T]))
    q, k = (torch.nn.functional.normalize(torch.randn(T, 1, d, generator=g), dim=-1) for _ in range(2))
    v, ab, state = torch.randn(T, dv, generator=g).to(DEV), torch.rand(T, 1, 4, generator=g), torch.randn(1, 1, dv, d, generator=g) * 0.3
    prep = torch.cat([q.reshape(T, -1), k.reshape(T, -1), ab.reshape(T, -1), torch.zeros(T, 8)], 1).to(DEV)
    runs = []
    for spoil in (False, True):
        if spoil:
            state[0, 0, col, row] = value
        after = state.to(DEV)
        runs.append((ops.gated_delta_rule(prep, v, after, slots, cu, pos, 1, 1, d, dv, per_head=True, max_q_len=T), after[0, 0]))
    others = [c for c in range(dv) if c != col]
    (clean, clean_s), (got, got_s) = runs
    assert torch.equal(got[:, others], clean[:, others]) and torch.equal(got_s[others], clean_s[others])
    if value == 3e38:      # the memory fades: finite, and of the size that the recurrence gives in float64
        want = _oracle(q, k, v.cpu().view(T, 1, dv), ab[:, :, 0], ab[:, :, 1], state, slots.cpu(), cu.cpu(), pos.cpu())
        for a, b in ((got[:, col].cpu(), want[0][:, 0, col]), (got_s[col].cpu(), want[1][0, 0, col])):
            assert a.isfinite().all() and (a.double() - b).abs().max() <= 2e-5 * b.abs().max()
    else:
        assert not got[:, col].isfinite().any() and not got_s[col].isfinite().any()


@pytest.mark.parametrize("d,dv,T", [(128, 128, 128), (68, 20, 65)])
def test_what_is_held_under_a_key_is_taken_off_to_the_last_bit(d, dv, T, monkeypatch):
    """Keys that are one place each, all different, without decay, written with nought at full strength: every product with the memory selects a
    row of it, which is nought afterwards, and the rows of no key stay what they are."""
    from pico_vllm_b200 import ops
    monkeypatch.setattr(ops, "delta_chunks_take", lambda *a: True)
    g = torch.Generator().manual_seed(T)
    cu, pos, slots = (t.to(DEV) for t in _segments([T]))
    at = torch.randperm(d, generator=g)[:T]
    k = torch.nn.functional.one_hot(at, d).float()
    state = torch.randn(1, 2, dv, d, generator=g)
    ab = torch.ones(T, 2, 4)
    prep = torch.cat([torch.randn(T, d, generator=g), k, ab.reshape(T, -1), torch.zeros(T, 8)], 1).to(DEV)
    after = state.to(DEV)
    ops.gated_delta_rule(prep, torch.zeros(T, 2 * dv, device=DEV), after, slots, cu, pos, 2, 1, d, dv, per_head=True, max_q_len=T)
    want = state.clone()
    want[..., at] = 0
    assert torch.equal(after.cpu(), want)
