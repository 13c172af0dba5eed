"""What the float32 products' own kernel may be given: tensors that are their numbers in memory and nothing else."""
import torch
from torch.autograd import forward_ad

from pico_vllm_b200 import ops


def test_tensors_that_are_only_numbers_in_memory():
    x = torch.randn(4, 8)
    assert ops._plain(x) and ops._plain(x[:, 1:]) and ops._plain(torch.nn.Parameter(x, requires_grad=False))
    assert not ops._plain(x.to_sparse()) and not ops._plain(torch._neg_view(x))
    assert not ops._plain(x.as_subclass(type("Own", (torch.Tensor,), {})))
    with forward_ad.dual_level():
        assert not ops._plain(forward_ad.make_dual(x, x)) and ops._plain(x)
    seen = []
    torch.func.vmap(lambda a: (seen.append(ops._nothing_follows()), a + 1)[1])(x)
    torch.func.grad(lambda a: (seen.append(ops._nothing_follows()), a.sum())[1])(x)
    torch.func.jvp(lambda a: (seen.append(ops._nothing_follows()), a.sum())[1], (x,), (x,))
    assert seen == [False] * 3


def test_fake_tensors_and_devices_without_kernels_are_the_library_s():
    from torch._subclasses import FakeTensorMode
    with FakeTensorMode():
        x, w = torch.empty(32, 1152, device="cuda"), torch.empty(512, 1152, device="cuda")
        assert not ops._plain(x) and not ops.f32_takes(x, w) and ops.linear(x, w).shape == (32, 512)
    x, w = torch.ones(32, 1152), torch.ones(512, 1152)
    assert ops._plain(x) and not ops.f32_takes(x, w)
