"""Checks of the native host path that come before anything is launched, so that they can be met without a GPU."""
import pytest
import torch

from omnimem_b200._lib import NSABackendError, host

NONE = (None, None)


def _bf16(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


@pytest.mark.parametrize("y", [_bf16(1, 4, 64), _bf16(2, 4, 32), torch.zeros(2, 4, 64)])
def test_residual_norm_refuses_another_residual(y):
    """The kernel reads x's rows from y: one that is smaller, or of another type, would be read past its end."""
    with pytest.raises(NSABackendError, match="y of shape|dtype"):
        host.residual_norm(_bf16(2, 4, 64), y, NONE, NONE, NONE, True, True, 1e-6)


@pytest.mark.parametrize("which", range(3))
@pytest.mark.parametrize("vec", [(_bf16(32), None), (_bf16(64, 2)[:, 0], None), (torch.zeros(64), None), (None, torch.zeros(32)),
                                 (None, _bf16(64)), (None, torch.zeros(64, 2)[:, 0])])
def test_residual_norm_refuses_other_vectors(which, vec):
    vecs = [NONE, NONE, NONE]
    vecs[which] = vec
    with pytest.raises(NSABackendError, match="contiguous values|dtype"):
        host.residual_norm(_bf16(2, 4, 64), _bf16(2, 4, 64), *vecs, True, True, 1e-6)


@pytest.mark.parametrize("w", [_bf16(32), torch.zeros(64), _bf16(64, 2)[:, 0]])
def test_norms_refuse_other_weights(w):
    with pytest.raises(NSABackendError, match="contiguous values|dtype"):
        host.rms_rows(_bf16(4, 64), w, 1e-6)
    rope = host.Rope(*(torch.zeros(8, n, 2, dtype=torch.float64) for n in (12, 10, 10)), 2, 2, 1, 1, 1, 0)
    for pair in ((w, _bf16(64)), (_bf16(64), w)):
        with pytest.raises(NSABackendError, match="contiguous values|dtype"):
            host.qk_norm_rope(_bf16(4, 64), _bf16(4, 64), *pair, 1e-6, 1, rope)


@pytest.mark.parametrize("k", [_bf16(2, 64), _bf16(4, 128), torch.zeros(4, 64)])
def test_query_norm_refuses_other_keys(k):
    rope = host.Rope(*(torch.zeros(8, n, 2, dtype=torch.float64) for n in (12, 10, 10)), 2, 2, 1, 1, 1, 0)
    with pytest.raises(NSABackendError, match="k of shape|dtype"):
        host.qk_norm_rope(_bf16(4, 64), k, _bf16(64), _bf16(64), 1e-6, 1, rope)


def test_rows_of_no_values_are_refused():
    with pytest.raises(NSABackendError, match="rows of shape"):
        host.residual_norm(_bf16(3, 0), None, NONE, NONE, NONE, True, True, 1e-6)
    with pytest.raises(NSABackendError, match="rows of shape"):
        host.rms_rows(_bf16(3, 0), _bf16(0), 1e-6)


def _row_views():
    """[..., 2, 3] views whose leading dimensions lie in every manner: contiguous, cut, spread, repeated, turned."""
    base = torch.arange(4000)
    yield base[:120].view(2, 10, 2, 3)
    yield base[:120].view(2, 1, 10, 2, 3)[:, :, :4]                      # the middle one says nothing
    yield base[:120].view(2, 1, 10, 2, 3)[:1, :, :4]
    yield base[:480].view(2, 10, 24)[..., 6:12].unflatten(-1, (2, 3))      # a view into a wider projection
    yield base[:480].view(4, 5, 24)[:, 1:2, 6:12].unflatten(-1, (2, 3))
    yield base[:24].view(4, 2, 3).expand(2, 1, 4, 2, 3)
    yield base[:6].view(1, 2, 3).expand(2, 4, 2, 3)
    yield base[:120].view(2, 10, 2, 3).transpose(0, 1)
    yield base[:6].view(1, 1, 2, 3)
    yield torch.as_strided(base, (3, 1, 4, 2, 3), (24, 24, 6, 3, 1))
    yield torch.as_strided(base, (3, 1, 4, 2, 3), (60, 60, 6, 3, 1))
    yield torch.as_strided(base, (3, 1, 4, 2, 3), (24, 999, 6, 3, 1))
    yield torch.as_strided(base, (3, 2, 1, 2, 3), (12, 6, 7, 3, 1))


def test_even_stride_finds_the_stride_of_rows_that_lie_evenly_and_no_other():
    for t in _row_views():
        dims, n = t.dim() - 2, t[..., 0, 0].numel()
        at = [int(x) for x in t[..., 0, 0].reshape(-1)]                    # (the values are their own positions)
        steps = {b - a for a, b in zip(at, at[1:])}
        got = host.even_stride(t, dims)
        assert (got is not None) == (len(steps) <= 1), (t.shape, t.stride(), got)
        if got is not None:
            assert [at[0] + i * got for i in range(n)] == at


@pytest.mark.parametrize("sizes", [(1, 64, 2), (1, 64, 2, 64, 2), (64,)])
def test_operators_refuse_other_ranks(sizes):
    """A fifth dimension used to be an error of the unpacking; the native path would read its first slice."""
    from omnimem_b200 import ops
    x, good, ids = _bf16(*sizes), _bf16(1, 64, 2, 64), torch.zeros(1, 1, 2, 1, dtype=torch.int32)
    mask = (64, 64, 64, 1, 0, 0, 0, False, False, False, 0, 1)
    calls = [lambda: ops.pool_rows(x, 4), lambda: host.topk(x, good, 1, 1.0, mask, False), lambda: host.topk(good, x, 1, 1.0, mask, False),
             lambda: host.select_blocks(x, good, 1, 1.0, mask, False), lambda: host.select_blocks(good, x, 1, 1.0, mask, False),
             lambda: ops.DenseKV(x, x)]
    for call in calls:
        with pytest.raises(ValueError, match="four dimensions"):
            call()


def test_same_bytes():
    a = torch.polar(torch.ones(6, 4, dtype=torch.float64), torch.arange(24, dtype=torch.float64).view(6, 4))
    assert host.same_bytes(a, a.clone()) and host.same_bytes(a[:0], a[:0].clone())
    last = a.clone()
    last[5, 3] += 1e-16j
    assert not any(host.same_bytes(a, b) for b in (last, a[:5], a.conj(), a.to(torch.complex64), a.t().contiguous().t(), a.view(4, 6)))


@pytest.mark.gpu
def test_gates_and_norms_of_views_equal_those_of_their_copies(dev):
    from omnimem_b200 import ops
    g = torch.Generator(device=dev).manual_seed(0)
    for view in _row_views():
        # the same view of random values
        logits = torch.randn(4000, generator=g, device=dev).to(torch.bfloat16).as_strided(view.shape, view.stride(), view.storage_offset())
        o = [torch.randn(*view.shape[:-1], 8, generator=g, device=dev).to(torch.bfloat16) for _ in range(3)]
        assert torch.equal(ops.gate_combine(logits, *o), ops.gate_combine(logits.contiguous(), *o))
        # rows of 16 values at the view's leading strides (16 bytes apart)
        lead, strides = view.shape[:-2], [s * 8 for s in view.stride()[:-2]]
        x = torch.randn(40000, generator=g, device=dev).to(torch.bfloat16).as_strided((*lead, 16), (*strides, 1))
        w = torch.randn(16, generator=g, device=dev).to(torch.bfloat16)
        assert torch.equal(host.rms_rows(x, w, 1e-6), host.rms_rows(x.contiguous(), w, 1e-6))


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1, 64, 2), (1, 64, 2, 64, 2)])
def test_attention_refuses_other_ranks(dev, sizes):
    from omnimem_b200 import ops
    good, x = (torch.zeros(*s, device=dev, dtype=torch.bfloat16) for s in ((1, 64, 2, 64), sizes))
    ids, lse = torch.zeros(1, 1, 2, 1, dtype=torch.int32, device=dev), torch.zeros(1, 2, 64, device=dev)
    kv = ops.DenseKV(good, good)
    ops.sel_fwd(good, kv, ids, 64, 1, 0.1, False, 64)
    for call in (lambda: ops.sel_fwd(x, kv, ids, 64, 1, 0.1, False, 64), lambda: ops.range_fwd(x, kv, 0, 1, 64, 0.1),
                 lambda: ops.sel_bwd(good, kv, ids, x, lse, good, 64, 1, 0.1, False, 64),
                 lambda: ops.sel_bwd(good, kv, ids, good, lse, x, 64, 1, 0.1, False, 64),
                 lambda: ops.sel_bwd(good, kv, ids[None], good, lse, good, 64, 1, 0.1, False, 64)):
        with pytest.raises((ValueError, RuntimeError)):
            call()
