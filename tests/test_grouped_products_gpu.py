"""One product per group of rows on the tcgen05 tensor cores: groups that are empty, of one row, of whole tiles and one more; widths that
end inside a tile; and dense products whose last tile is short."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _silu_mul(y, limit):
    g, u = y.chunk(2, -1)
    if limit:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    return g * torch.sigmoid(g) * u


@pytest.mark.parametrize("counts", [[1], [0, 256, 0, 1, 257, 0], [512, 513, 128, 0, 300], [0, 0, 5], [40] * 40, [1030, 129], [3] * 70 + [600]])
@pytest.mark.parametrize("N,K", [(256, 64), (272, 200), (1552, 136)])
@pytest.mark.parametrize("epi,limit", [(0, 0.0), (2, 0.0), (3, 1.5)])
@pytest.mark.parametrize("rows", [0, -1, 64, 320, 512])
def test_groups(counts, N, K, epi, limit, rows):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(sum(counts) + N)
    E, n = len(counts), sum(counts)
    x = torch.randn(n + 3, K, generator=g, device=DEV).bfloat16()[:n]
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    c = torch.tensor(counts)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), c.cumsum(0)]).to(torch.int32).to(DEV)
    cols = N if epi == 0 else N // 2
    out = torch.full((n + 2, cols), float("nan"), dtype=torch.bfloat16, device=DEV)
    lib = ops.library()
    assert lib.pico_gemm_tcgen05_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), offsets.data_ptr(), n, E, N, K, epi, rows,
                                         limit, ops._stream()) == 0
    at = 0
    for e, k in enumerate(counts):
        y = x[at:at + k].float() @ w[e].float().t()
        want = y if epi == 0 else _silu_mul(y, limit)
        got = out[at:at + k].float()
        # one rounding to 16 bits of a float32 sum of K products of order K^-1/2
        assert torch.allclose(got, want, atol=2e-2, rtol=1e-2), (e, float((got - want).abs().max()))
        at += k
    assert torch.isnan(out[n:].float()).all()
    assert ops.tc_status() == 0


@pytest.mark.parametrize("M", [512, 513, 640, 768, 769, 1025, 2111])
def test_a_short_last_tile_of_a_dense_product(M):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    K, I = 328, 1000
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(2 * I, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    y = x.float() @ w.float().t()
    for rows in (256, 512):
        assert torch.allclose(ops.tc_linear(x, w, rows=rows).float(), y, atol=2e-2, rtol=1e-2)
        assert torch.allclose(ops.tc_gate_up_swiglu(x, w, rows=rows).float(), _silu_mul(y, 0.0), atol=2e-2, rtol=1e-2)
        res = torch.ones(M, 2 * I, device=DEV)
        ops.tc_linear_residual(x, w, res, rows=rows)
        assert torch.allclose(res, y + 1, atol=1e-3, rtol=1e-3)
    assert ops.tc_status() == 0


@pytest.mark.parametrize("counts", [[1, 0, 32, 33], [300, 0, 64, 65, 513, 2], [31, 64, 250] * 30])
@pytest.mark.parametrize("N", [352, 4480])           # gate halves of 176 and 2,240: multiples of 16 that end inside a tile of 128
@pytest.mark.parametrize("epi", [0, 2])
@pytest.mark.parametrize("rows", [0, -1, 512])
def test_long_rows_go_around_the_stages(counts, N, epi, rows):
    """16 blocks of K: every stage is filled again and again, by short tiles after long ones and the other way round."""
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(sum(counts) + N)
    n, E, K = sum(counts), len(counts), 1000
    x = torch.randn(n, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    offsets = torch.tensor([0] + counts, device=DEV).cumsum(0).to(torch.int32)
    out = torch.empty(n, N if epi == 0 else N // 2, dtype=torch.bfloat16, device=DEV)
    assert ops.library().pico_gemm_tcgen05_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), offsets.data_ptr(), n, E, N, K, epi, rows,
                                                   0.0, ops._stream()) == 0
    y = torch.cat([a.float() @ w[e].float().t() for e, a in enumerate(x.split(counts))])
    assert torch.allclose(out.float(), y if epi == 0 else _silu_mul(y, 0.0), atol=2e-2, rtol=1e-2)
    assert ops.tc_status() == 0


@pytest.mark.parametrize("N,K", [(16, 16), (48, 24), (352, 48), (272, 56)])
@pytest.mark.parametrize("epi", [0, 2])
@pytest.mark.parametrize("rows", [0, -1, 64])
def test_products_narrower_than_a_block_of_k(N, K, epi, rows):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N + K)
    counts = [0, 270, 1, 33, 700]
    n, E = sum(counts), len(counts)
    x = torch.randn(n, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    offsets = torch.tensor([0] + counts, device=DEV).cumsum(0).to(torch.int32)
    out = torch.empty(n, N if epi == 0 else N // 2, dtype=torch.bfloat16, device=DEV)
    assert ops.library().pico_gemm_tcgen05_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), offsets.data_ptr(), n, E, N, K, epi, rows,
                                                   0.0, ops._stream()) == 0
    y = torch.cat([a.float() @ w[e].float().t() for e, a in enumerate(x.split(counts))])
    assert torch.allclose(out.float(), y if epi == 0 else _silu_mul(y, 0.0), atol=2e-2, rtol=1e-2)
    assert ops.tc_status() == 0


@pytest.mark.parametrize("E", [513, 1024])
@pytest.mark.parametrize("epi,N", [(0, 72), (2, 96)])
@pytest.mark.parametrize("rows", [0, -1, 64])
def test_hundreds_of_groups(E, epi, N, rows):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(E + N)
    counts = [(7 * e) % 5 for e in range(E)]
    counts[1], counts[-1] = 300, 70
    n, K = sum(counts), 136
    x = torch.randn(n, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    expert = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).to(DEV)
    offsets = torch.tensor([0] + counts, device=DEV).cumsum(0).to(torch.int32)
    out = torch.empty(n, N if epi == 0 else N // 2, dtype=torch.bfloat16, device=DEV)
    assert ops.library().pico_gemm_tcgen05_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), offsets.data_ptr(), n, E, N, K, epi, rows,
                                                   0.0, ops._stream()) == 0
    y = torch.bmm(w.float()[expert], x.float()[:, :, None])[:, :, 0]
    assert torch.allclose(out.float(), y if epi == 0 else _silu_mul(y, 0.0), atol=2e-2, rtol=1e-2)
    assert ops.tc_status() == 0


FORMS = {"gated": dict(), "capped": dict(act="capped", limit=0.9), "weight in": dict(gated=False, act="relu2", weight_on_input=True),
         "weight out": dict(gated=False, act="silu")}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("T", [35, 640])             # on either side of 245 rows an expert on average, with five experts of which one gets nothing
@pytest.mark.parametrize("D,ff", [(64, 64), (72, 104), (136, 112)])
@pytest.mark.parametrize("identity,base", [(0, False), (2, True)])
def test_experts_through_the_tensor_cores(form, T, D, ff, identity, base):
    """Listing, gathering, both products with what lies between them and the placed sum, against the sum in float64."""
    from pico_vllm_b200 import ops
    how = dict(FORMS[form])
    if identity and how.get("weight_on_input"):
        pytest.skip("experts that pass their input on take their weight on the output")
    how["act"] = {"capped": ops.MOE_ACT_CAPPED, "relu2": ops.MOE_ACT_RELU2}.get(how.get("act"), ops.MOE_ACT_SILU)
    gated, limit = how.get("gated", True), how.get("limit", 0.0)
    E, top = 5, 3
    g = torch.Generator(device=DEV).manual_seed(T + D + ff)
    h = torch.randn(T, D, generator=g, device=DEV).bfloat16()
    up = (torch.randn(E, (2 if gated else 1) * ff, D, generator=g, device=DEV) * D ** -0.5).bfloat16()
    down = (torch.randn(E, D, ff, generator=g, device=DEV) * ff ** -0.5).bfloat16()
    keys = torch.rand(T, E + identity, generator=g, device=DEV)
    keys[:, 3] = -1.0                                                # nobody asks for expert 3
    idx = keys.topk(top, -1).indices.to(torch.int32).contiguous()
    wgt = torch.softmax(torch.randn(T, top, generator=g, device=DEV), -1)
    add = torch.randn(T, D, generator=g, device=DEV).bfloat16() if base else None
    assert ops.moe_tc_takes(h, up, down, T * top)
    y = ops.moe_experts(h, idx, wgt, up, down, base=add, identity=identity, **how).double()
    want = add.double().clone() if base else torch.zeros(T, D, dtype=torch.float64, device=DEV)
    x = h.double()
    for e in range(E + identity):
        w = (wgt.double() * (idx == e)).sum(-1, keepdim=True)
        if e >= E:
            want += w * x
            continue
        z = x @ up[e].double().t()
        if gated:
            a = _silu_mul(z, limit)
        else:
            z = z * w if how.get("weight_on_input") else z
            a = z.clamp(min=0) ** 2 if how["act"] == ops.MOE_ACT_RELU2 else z * torch.sigmoid(z)
        o = a @ down[e].double().t()
        want += o * (idx == e).any(-1, keepdim=True) if how.get("weight_on_input") else o * w
    # bfloat16 keeps 2^-9 of a number: once between the products (and once before the activation where there is no gate), once after the
    # second, once for the sum
    assert float((y - want).abs().max()) <= 2 ** -7 * float(want.abs().max())
    assert ops.tc_status() == 0
