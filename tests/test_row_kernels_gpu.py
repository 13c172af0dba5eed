"""Kernels that read a row four numbers at a time beside their general forms: the short convolution, the norm in groups, the inputs
of the delta rule; and the router and the lists of tokens per expert."""
import pytest
import torch

import fake_ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F32, BF16 = torch.float32, torch.bfloat16


def _close(got, want, tol, what):
    # tol: of the larger of one and the value; float32 sums of some hundreds of products, or one rounding to 16 bits
    off = (got.float().cpu() - want.float()).abs() / want.float().abs().clamp(min=1.0)
    assert float(off.max()) <= tol, (what, float(off.max()))


def _segments(lens, pad_at=None):
    cu, pos, seg = [0], [], []
    for s, n in enumerate(lens):
        cu.append(cu[-1] + n)
        pos += [-1] * n if s == pad_at else list(range(5 * s, 5 * s + n))
        seg += [s] * n
    i32 = lambda v: torch.tensor(v, dtype=torch.int32)
    return i32(cu), i32(pos), i32(seg), i32(list(range(len(lens) - 1, -1, -1)))


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("C,off", [(8, 4), (1032, 0), (12, 2), (9, 0)])
@pytest.mark.parametrize("taps", [1, 2, 4])
@pytest.mark.parametrize("lens,pad_at", [([257], None), ([1, 2, 250, 3, 1, 8, 1, 64], 3)])
def test_short_convolution(dtype, C, off, taps, lens, pad_at):
    from pico_vllm_b200 import ops
    g = torch.Generator().manual_seed(C + taps)
    cu, pos, seg, slots = _segments(lens, pad_at)
    T, S = int(cu[-1]), len(lens)
    proj = torch.randn(T, C + 8, generator=g).to(dtype)
    w, b = torch.randn(C, taps, generator=g), torch.randn(C, generator=g)
    state = torch.randn(S + 1, taps - 1, C, generator=g)
    got_state = state.to(DEV)
    for bias in (b, None):
        want = fake_ops.causal_conv_silu(proj, off, w, bias, state, seg, slots, cu, pos)
        got = ops.causal_conv_silu(proj.to(DEV), off, w.to(DEV), None if bias is None else bias.to(DEV), got_state, seg.to(DEV),
                                   slots.to(DEV), cu.to(DEV), pos.to(DEV))
        _close(got, want, 1e-5, "convolution")
        if taps > 1:
            _close(got_state, state, 1e-6, "state")


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("groups,n", [(12, 128), (5, 4), (1, 508), (3, 132), (4, 130)])
def test_group_norm(dtype, groups, n):
    from pico_vllm_b200 import ops
    g = torch.Generator().manual_seed(n)
    x = torch.randn(9, groups * (n + 4), generator=g)
    w = torch.rand(groups * n, generator=g) + 0.5
    gate = (torch.randn(9, groups * n + 8, generator=g) * 3).to(dtype)
    for act, gt in (("sigmoid", gate[:, 8:]), ("silu", gate[:, 4:4 + groups * n]), ("silu", gate[:, 1:1 + groups * n]), ("silu", None)):
        want = fake_ops.group_rms_norm(x, groups, n, n + 4, w, 1e-5, dtype, post_gate=gt, post_act=act)
        on_gpu = None if gt is None else gate.to(DEV)[:, gt.storage_offset():gt.storage_offset() + groups * n]
        got = ops.group_rms_norm(x.to(DEV), groups, n, n + 4, w.to(DEV), 1e-5, dtype, post_gate=on_gpu, post_act=act)
        _close(got, want, 2e-6 if dtype == F32 else 1e-2, act)


@pytest.mark.parametrize("H,G,d", [(4, 2, 16), (12, 6, 128), (3, 1, 100), (2, 2, 132), (2, 1, 30)])
@pytest.mark.parametrize("longest", [1, 8])
def test_delta_inputs(H, G, d, longest):
    from pico_vllm_b200 import ops
    g = torch.Generator().manual_seed(d)
    T = 11
    xc = torch.randn(T, 2 * G * d + 12, generator=g)
    proj = torch.randn(T, 2 * H + 4, generator=g) * 2
    dt_bias, a_log = torch.randn(H, generator=g), torch.randn(H, generator=g) - 1.0
    want = fake_ops.delta_prepare(xc, 4, 4 + G * d, proj, 2, proj[:, 2 + H:2 + 2 * H], dt_bias, a_log, H, G, d, per_head=True, max_q_len=longest)
    p = proj.to(DEV)
    got = ops.delta_prepare(xc.to(DEV), 4, 4 + G * d, p, 2, p[:, 2 + H:2 + 2 * H], dt_bias.to(DEV), a_log.to(DEV), H, G, d, per_head=True,
                            max_q_len=longest).cpu()
    pair, dots = got[:, 2 * G * d:2 * G * d + 4 * H].view(T, H, 4), got[:, 2 * G * d + 4 * H:].view(T, G, 8)
    pair[:, :, 2:] = 0                             # numbers nobody reads
    dots[:, :, 7 if longest >= ops.DELTA_BLOCK_MIN_TOKENS else 1:] = 0
    _close(got, want, 2e-6, "delta_prepare")


def test_delta_inputs_whose_squares_overflow():
    """A query and a key of 1e20, whose sums of squares are infinite: both come out as nought, and so does their dot product."""
    from pico_vllm_b200 import ops
    H, G, d, T = 2, 2, 128, 3
    xc, proj, zero = torch.ones(T, 2 * G * d, device=DEV), torch.zeros(T, 2 * H, device=DEV), torch.zeros(H, device=DEV)
    xc[1] = 1e20
    got = ops.delta_prepare(xc, 0, G * d, proj, 0, proj[:, H:], zero, zero, H, G, d, per_head=True)
    assert not got[1, :2 * G * d].any() and not got[1, 2 * G * d + 4 * H::8].any()
    assert got[[0, 2], 2 * G * d + 4 * H].gt(0).all()


@pytest.mark.parametrize("T,E,top", [(1, 1, 1), (5, 16, 4), (33, 3, 2), (2050, 16, 4), (700, 130, 32), (64, 4096, 8)])
def test_lists_of_tokens_per_expert(T, E, top):
    from pico_vllm_b200 import ops
    g = torch.Generator().manual_seed(E)
    n = T * top
    idx = torch.randint(0, max(1, E - 1), (n,), generator=g).to(torch.int32)          # the last expert gets none
    bm = (16, 64)[T % 2]
    out = [torch.full((k,), -1, dtype=torch.int32, device=DEV) for k in (E + 1, E + 1, n, n)]
    lib = ops.library()
    dev = idx.to(DEV)
    assert lib.pico_moe_group(dev.data_ptr(), n, E, bm, *[t.data_ptr() for t in out], ops._stream()) == 0
    offsets, tiles, perm, place = [t.cpu().long() for t in out]
    counts = torch.bincount(idx.long(), minlength=E)
    assert offsets.tolist() == [0] + counts.cumsum(0).tolist()
    assert tiles.tolist() == [0] + (-(-counts // bm)).cumsum(0).tolist()
    assert idx.long()[perm].tolist() == idx.long().sort().values.tolist()        # (the order inside a list is left open)
    assert torch.equal(perm[place], torch.arange(n))


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("T,D,E", [(1030, 64, 5), (1025, 1536, 16), (1024, 3000, 8), (515, 72, 40), (9, 64, 16), (1030, 30, 5)])
def test_router(dtype, T, D, E):
    from pico_vllm_b200 import ops
    g = torch.Generator().manual_seed(T + D)
    top = 3
    h, w, b = torch.randn(T, D, generator=g).to(dtype), torch.randn(E, D, generator=g), torch.randn(E, generator=g)
    got_i, got_w = ops.moe_route(h.to(DEV), w.to(DEV), b.to(DEV), top)
    z = h.double() @ w.double().t() + b.double()
    order = z.sort(-1, descending=True).values
    clear = (order[:, :top] - order[:, 1:top + 1]).min(-1).values > 1e-3 * D ** 0.5     # (choices that a rounding cannot turn)
    top_z, top_i = z.topk(top, -1)
    assert clear.float().mean() > 0.9 and torch.equal(got_i.cpu().long()[clear], top_i[clear])
    _close(got_w.cpu()[clear], torch.softmax(top_z, -1)[clear], 1e-4, "weights")
