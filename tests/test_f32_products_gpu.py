"""float32 products as three tf32 products on the tensor cores against float64: the edges of tiles, of the 32-wide pieces of K and of its
parts, rows that lie apart, and sums that are no number."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K", [(17, 512, 1024), (16, 132, 36), (1, 4, 4), (33, 516, 1028), (128, 128, 1536), (129, 260, 1540), (340, 2048, 1536),
                                   (2049, 640, 1024), (100, 1536, 8960), (64, 20000, 1024)])
@pytest.mark.parametrize("apart", [0, 4])
def test_against_float64(M, N, K, apart):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    wide = torch.randn(M, K + apart, device=DEV, generator=g)
    x, w = wide[:, :K], torch.randn(N, K, device=DEV, generator=g) * 0.02
    got, want, size = ops.linear_f32(x, w).double(), x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    # of each product: 2^-24 for what either splitting leaves and for the product of the small parts; of a sum: one cut of 2^-23 for each of the
    # eight instructions of 64 terms, then a rounding of 2^-24 for each 64 terms and each part of K
    bound = (3 + 16 + K / 64 + 40) * 2.0 ** -24
    assert float(((got - want).abs() / size.clamp_min(1e-30)).max()) <= bound
    # and no further off than float32 multiply-adds, as a whole
    if M >= 17 and K >= 1024:
        plain = torch.mm(x, w.t()).double()
        assert float((got - want).norm()) <= 1.05 * float((plain - want).norm())
    assert ops.tf_status() == 0


@pytest.mark.parametrize("M,N,K", [(40, 132, 64), (40, 512, 1024)])
def test_sums_that_are_no_number_are_what_float32_gives(M, N, K):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g)
    clean = ops.linear_f32(x, w)
    x[3, 5], x[7, 1], w[9, 2], w[10, 2], x[11, 3] = float("inf"), float("nan"), 3e37, float("-inf"), 3e38
    got, plain = ops.linear_f32(x, w), x.double() @ w.double().t()
    plain = torch.where(plain.abs() > 3.4028235e38, plain.sign() * float("inf"), plain)
    assert torch.equal(got.isnan(), plain.isnan())
    sure = plain.abs() < 3e38                                   # (a sum may pass the largest number on its way to a smaller one)
    assert torch.equal(got.isinf() & ~sure, plain.isinf() & ~sure & got.isinf())
    ok = plain.isfinite() & got.isfinite()
    assert float(((got.double() - plain).abs() / (x.double().abs() @ w.double().abs().t()))[ok].max()) <= 100 * 2.0 ** -24
    rows = [i for i in range(M) if i not in (3, 7, 11)]
    cols = [i for i in range(N) if i not in (9, 10)]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


@pytest.mark.parametrize("M,N,K,off,takes", [(16, 2048, 1536, 0, False), (17, 2048, 1536, 0, True), (17, 508, 1536, 0, False), (17, 512, 1020, 0, False),
                                             (17, 512, 1026, 0, False), (17, 514, 1024, 0, False), (17, 512, 1024, 1, False), (17, 512, 1024, 4, True),
                                             (32, 32000, 1024, 0, False), (33, 32000, 1024, 0, True)])
def test_which_products_go_there(M, N, K, off, takes):
    from pico_vllm_b200 import ops
    x, w = torch.ones(M, K + off, device=DEV)[:, off:], torch.ones(N, K, device=DEV)
    assert ops.f32_takes(x, w) == takes
    before = ops.launches
    assert bool((ops.linear(x, w) == K).all())
    assert (ops.launches > before) == takes
    if M == 17 and takes:
        assert not ops.f32_takes(torch.ones(1, K, device=DEV).expand(M, K), w) and not ops.f32_takes(x, torch.ones(K, N, device=DEV).t())


def test_a_product_with_a_gradient_is_the_library_s_and_a_wait_that_ran_out_is_seen(monkeypatch):
    from pico_vllm_b200 import ops
    x, w = torch.ones(32, 1024, device=DEV, requires_grad=True), torch.ones(512, 1024, device=DEV)
    ops.linear(x, w).sum().backward()
    assert bool((x.grad == 512).all())
    assert ops.tc_status() == 0
    monkeypatch.setattr(ops, "tf_status", lambda: 1)
    assert ops.tc_status() == 1
