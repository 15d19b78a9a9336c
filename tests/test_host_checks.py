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
