"""The differentiable operators as autograd sees them: errors of their backward, and the transforms that look at a Function."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(dev, dtype=torch.bfloat16):
    g = torch.Generator(device=dev).manual_seed(0)
    q, k, v = (torch.randn(1, 128, 2, 128, generator=g, device=dev).to(dtype).requires_grad_(True) for _ in range(3))
    return q, k, v, torch.tensor([0, 1], dtype=torch.int32, device=dev).expand(1, 2, 2, 2).contiguous()


def _attend(q, k, v, ids):
    from omnimem_b200.nsa.ops import selection_attention
    return selection_attention(q, k, v, ids, 2, 64, group_size=64)


def test_errors_of_a_backward_are_the_packages_own(dev):
    from omnimem_b200._lib import NSABackendError
    from omnimem_b200.nsa.ops import gated_branch_sum
    logits = torch.zeros(1, 4, 2, 3, device=dev, dtype=torch.bfloat16, requires_grad=True)
    branch = torch.ones(1, 4, 2, 24, device=dev, dtype=torch.bfloat16)      # a head dim that only the forward is built for
    x = gated_branch_sum(logits, branch, branch, branch)
    for _ in range(2):
        with pytest.raises(NSABackendError, match="head dim 24"):
            x.sum().backward(retain_graph=True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t):      # comes back on the CPU
        out = _attend(*_inputs(dev))
    with pytest.raises(NSABackendError, match="CUDA tensors"):
        out.sum().backward()


def test_saved_tensor_hooks_see_the_saved_tensors(dev):
    want = torch.autograd.grad(_attend(*(a := _inputs(dev))).sum(), a[:3])
    with torch.autograd.graph.save_on_cpu():
        out = _attend(*(b := _inputs(dev)))
    assert all(map(torch.equal, torch.autograd.grad(out.sum(), b[:3]), want))
