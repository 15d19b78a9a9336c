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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_the_autograd_function(dev, dtype):
    """SelectionAttentionB200 is a Function that can be applied and derived from; the native operator gives its results."""
    from omnimem_b200.nsa.ops.selection import SelectionAttentionB200
    assert issubclass(SelectionAttentionB200, torch.autograd.Function)

    class Doubled(SelectionAttentionB200):
        @staticmethod
        def forward(ctx, *args):
            return 2 * SelectionAttentionB200.forward(ctx, *args)

    *leaves, ids = _inputs(dev, dtype)
    native = _attend(*leaves, ids)
    out, lse = SelectionAttentionB200.apply(*leaves, ids, 64, 1, None, False, True, 64)
    assert torch.equal(out, native) and not lse.requires_grad and out.dtype == dtype
    up = torch.randn_like(out)
    want = torch.autograd.grad(native, leaves, up)
    assert all(map(torch.equal, torch.autograd.grad(out, leaves, up), want))
    assert torch.equal(Doubled.apply(*leaves, ids, 64, 1, None, False, False, 64), 2 * native)


def _gate(dev):
    from omnimem_b200.nsa.ops import gated_branch_sum
    g = torch.Generator(device=dev).manual_seed(1)
    args = [torch.randn(1, 8, 2, n, generator=g, device=dev).to(torch.bfloat16) for n in (3, 64, 64, 64)]
    return gated_branch_sum, args


def test_traces_compute_what_was_traced(dev):
    import warnings
    q, k, v, ids = (t.detach() for t in _inputs(dev))
    q2 = torch.randn_like(q)
    gate, args = _gate(dev)
    args2 = [torch.randn_like(t) for t in args]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")                                   # the id check reads values
        attend = torch.jit.trace(lambda a, b, c: _attend(a, b, c, ids), (q, k, v), check_trace=False)
        gated = torch.jit.trace(lambda *a: gate(*a), args, check_trace=False)
    junk = [torch.full_like(q, float("nan")) for _ in range(8)]           # what a fresh output would hold
    del junk
    assert torch.equal(attend(q2, k, v), _attend(q2, k, v, ids)) and torch.equal(gated(*args2), gate(*args2))


def test_transforms_are_refused(dev):
    """Not supported before the native operators, and not answered wrongly by them."""
    q, k, v, ids = (t.detach() for t in _inputs(dev))
    gate, args = _gate(dev)
    many = lambda t: torch.stack([t, t])
    for call in (lambda: torch.func.grad(lambda a: _attend(a, k, v, ids).sum())(q), lambda: torch.vmap(lambda a: _attend(a, k, v, ids))(many(q)),
                 lambda: torch.func.jvp(lambda a: _attend(a, k, v, ids), (q,), (q,)), lambda: torch.func.grad(lambda a: gate(a, *args[1:]).sum())(args[0]),
                 lambda: torch.vmap(lambda a: gate(a, *args[1:]))(many(args[0]))):
        with pytest.raises(RuntimeError):
            call()
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual
        for call in (lambda: _attend(dual(q, q), k, v, ids), lambda: gate(dual(args[0], args[0]), *args[1:])):
            with pytest.raises((RuntimeError, NotImplementedError)):
                call()
