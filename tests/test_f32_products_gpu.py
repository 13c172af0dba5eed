"""float32 products of three bfloat16 parts a factor on the tensor cores against float64: the edges of tiles, of the 32-wide pieces of K and
of its parts, rows that lie apart, sums of few terms and of terms of one sign, and sums that are no number."""
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
    assert float(((got - want).abs() / size.clamp_min(1e-30)).max()) <= _bound(M, N, K)
    # and no further off than float32 multiply-adds, as a whole
    if M >= 17 and K >= 1024:
        plain = torch.mm(x, w.t()).double()
        assert float((got - want).norm()) <= float((plain - want).norm())
    assert ops.tf_status() == 0


def _bound(M, N, K):
    """Largest error over the sum of the terms' sizes, in units of 2^-24.  Of each product 2^-6 (the c c that is left out, 2^-30).  Of 64 terms: the
    four instructions of the products a a cut off at most a unit of float32's last place each (2 units), and a rounding adds their sum to the others'.
    Of sixteen terms: the two instructions of a b and b a cut off the same of sums below 2^-6, the five others of sums below 2^-12.  Then a rounding
    for each part of K in both sums, and two of what is added at the end."""
    from pico_vllm_b200 import ops
    return (2 ** -6 + 4 * 2 - (-K // 64) - (-K // 16) * (2 * 2 * 2 ** -6 + 5 * 2 * 2 ** -12) + 1.1 * ops.library().pico_gemm_f32_parts(M, N, K) + 2) * 2.0 ** -24


def _few(M, K, n, g):
    """Rows with n numbers that are not nought."""
    x = torch.zeros(M, K, device=DEV)
    at = torch.rand(M, K, device=DEV, generator=g).topk(n, 1).indices
    return x.scatter_(1, at, torch.randn(M, n, device=DEV, generator=g))


@pytest.mark.parametrize("M,N,K", [(17, 512, 1024), (40, 640, 1540), (340, 2048, 1536)])
def test_rows_that_select_give_the_weights_bit_for_bit(M, N, K):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(K)
    w, at = torch.randn(N, K, device=DEV, generator=g), torch.randint(0, K, (M,), device=DEV, generator=g)
    x = torch.zeros(M, K, device=DEV).scatter_(1, at[:, None], 1.0)
    assert torch.equal(ops.linear_f32(x, w), w.t()[at])
    # and rows of w that select
    x, at = torch.randn(M, K, device=DEV, generator=g), torch.randint(0, K, (N,), device=DEV, generator=g)
    w = torch.zeros(N, K, device=DEV).scatter_(1, at[:, None], 1.0)
    assert torch.equal(ops.linear_f32(x, w), x[:, at])


@pytest.mark.parametrize("M,N,K", [(17, 512, 1024), (128, 640, 2052), (340, 2048, 1536)])
@pytest.mark.parametrize("kind", ["1", "2", "3", "8", "positive", "positive and few", "of all sizes", "one term dominates", "equal factors"])
def test_sums_of_few_terms_of_one_sign_and_of_all_sizes(M, N, K, kind):
    """Within the bound at every place, and as a whole no further from float64 than float32 multiply-adds."""
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + K)
    w = torch.randn(N, K, device=DEV, generator=g)
    if kind.isdigit():
        x = _few(M, K, int(kind), g)
    elif kind == "positive":
        x, w = 1 + torch.rand(M, K, device=DEV, generator=g), 1 + torch.rand(N, K, device=DEV, generator=g)
    elif kind == "positive and few":
        x, w = _few(M, K, 4, g).abs(), w.abs()
    elif kind == "of all sizes":
        x, w = (t * torch.exp2(40 * torch.rand(t.shape, device=DEV, generator=g) - 20) for t in (torch.randn(M, K, device=DEV, generator=g), w))
    elif kind == "one term dominates":
        x = torch.randn(M, K, device=DEV, generator=g) * 1e-3 + 30 * _few(M, K, 1, g)
    else:       # factors whose first eleven digits leave as much as they can
        x, w = torch.full((M, K), 1 + 2.0 ** -11 - 2.0 ** -23, device=DEV), torch.full((N, K), 1 + 2.0 ** -11 - 2.0 ** -23, device=DEV)
    got, want, size = ops.linear_f32(x, w).double(), x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert float(((got - want).abs() / size.clamp_min(1e-300)).max()) <= _bound(M, N, K)
    plain = torch.mm(x, w.t()).double()
    # (a single term's product is exact to 2^-28 before it is rounded)
    assert kind == "equal factors" or float((got - want).norm()) <= float((plain - want).norm()) + 2.0 ** -28 * float(want.norm())


@pytest.mark.parametrize("scale", [2.0 ** -100, 2.0 ** 100, 2.0 ** 126])
def test_very_small_and_very_large_numbers(scale):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(9)
    x, w = (torch.randn(*s, device=DEV, generator=g).clamp(-1, 1) for s in ((40, 1024), (512, 1024)))
    x, w = x * scale, w / 1024
    got, want = ops.linear_f32(x, w).double(), x.double() @ w.double().t()
    assert float((got - want).norm()) <= float((torch.mm(x, w.t()).double() - want).norm())


@pytest.mark.parametrize("M,N,K", [(40, 132, 64), (40, 512, 1024)])
def test_sums_that_are_no_number_are_what_float32_gives(M, N, K):
    from pico_vllm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g)
    clean = ops.linear_f32(x, w)
    x[3, 5], x[7, 1], w[9, 2], w[10, 2], x[11, 3] = float("inf"), float("nan"), 3e37, float("-inf"), 3e38
    got, plain = ops.linear_f32(x, w).double(), x.double() @ w.double().t()
    assert torch.equal(got.isnan(), plain.isnan())
    # infinities of an operand, with their signs
    assert plain[3].isinf().any() and plain[:, 10].isinf().any()
    assert torch.equal(got[plain.isinf()], plain[plain.isinf()])
    # and of finite numbers' sums, each with one large term at most that decides: no infinity below the largest number, none missing above it
    top = 3.4028235e38
    over, under = plain.isfinite() & (plain.abs() > 1.01 * top), plain.abs() < 0.99 * top
    assert over.any() and torch.equal(got[over], plain[over].sign() * float("inf"))
    assert float(((got - plain).abs() / (x.double().abs() @ w.double().abs().t()))[under].max()) <= _bound(M, N, K)
    rows = [i for i in range(M) if i not in (3, 7, 11)]
    cols = [i for i in range(N) if i not in (9, 10)]
    assert torch.equal(got[rows][:, cols], clean.double()[rows][:, cols])


@pytest.mark.parametrize("M,N,K,off,takes", [(16, 2048, 1536, 0, False), (17, 2048, 1536, 0, True), (17, 508, 1536, 0, False), (17, 512, 1020, 0, False),
                                             (17, 512, 1154, 0, False), (17, 514, 1152, 0, False), (17, 512, 1152, 1, False), (17, 512, 1152, 4, True),
                                             (17, 512, 1148, 0, False), (17, 2044, 1024, 0, False), (17, 2048, 1024, 0, True), (33, 1020, 1024, 0, False),
                                             (33, 1024, 1024, 0, True), (65, 636, 1024, 0, False), (65, 640, 1024, 0, True), (97, 512, 1024, 0, True),
                                             (32, 8192, 1024, 0, True), (32, 8196, 1024, 0, False), (32, 18944, 3584, 0, True), (32, 18948, 3584, 0, False),
                                             (32, 18944, 3580, 0, False), (33, 32000, 1024, 0, True)])
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
    x, w = torch.ones(32, 1152, device=DEV, requires_grad=True), torch.ones(512, 1152, device=DEV)
    ops.linear(x, w).sum().backward()
    assert bool((x.grad == 512).all())
    assert ops.tc_status() == 0
    monkeypatch.setattr(ops, "tf_status", lambda: 1)
    assert ops.tc_status() == 1


def test_what_is_more_than_numbers_in_memory_is_the_library_s():
    from torch.autograd import forward_ad
    from torch.utils.flop_counter import FlopCounterMode
    from pico_vllm_b200 import ops
    x, w = torch.ones(32, 1152, device=DEV), torch.ones(512, 1152, device=DEV)
    with forward_ad.dual_level():
        out = forward_ad.unpack_dual(ops.linear(forward_ad.make_dual(x, x), w))
        assert bool((out.primal == 1152).all()) and bool((out.tangent == 1152).all())
    assert bool((torch.func.vmap(lambda a: ops.linear(a, w))(x.expand(2, 32, 1152)) == 1152).all())
    assert bool((torch.func.grad(lambda a: ops.linear(a, w).sum())(x) == 512).all())
    assert bool((ops.linear(torch._neg_view(x), w) == -1152).all())
    with FlopCounterMode(display=False) as flops:
        ops.linear(x, w)
    assert flops.get_total_flops() == 2 * 32 * 512 * 1152
    assert ops.f32_takes(x, w) and ops.f32_takes(x, torch.nn.Parameter(w, requires_grad=False))
    with pytest.raises(RuntimeError):
        ops.linear(x, torch.ones(512, 1156, device=DEV))


def test_under_autocast_a_product_is_what_it_was():
    from pico_vllm_b200 import ops
    x, w = torch.randn(32, 1152, device=DEV), torch.randn(512, 1152, device=DEV)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got, plain = ops.linear(x, w), torch.mm(x, w.t())
    assert got.dtype == plain.dtype and torch.equal(got, plain)


def test_without_room_for_its_parts_a_product_is_the_library_s(monkeypatch):
    from pico_vllm_b200 import ops
    x, w = torch.randn(40, 2048, device=DEV), torch.randn(512, 2048, device=DEV)
    assert ops.library().pico_gemm_f32_parts(40, 512, 2048) > 1
    real, asked = torch.Tensor.new_empty, []

    def new_empty(self, size, *rest):
        if isinstance(size, int):
            asked.append(size)
            raise torch.OutOfMemoryError("no room")
        return real(self, size, *rest)
    monkeypatch.setattr(torch.Tensor, "new_empty", new_empty)
    got = ops.linear(x, w)
    assert len(asked) == 1 and torch.equal(got, torch.mm(x, w.t()))
