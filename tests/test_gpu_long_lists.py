"""Lists longer than shared memory would hold with an entry per tile or a ring per warp, mostly padding, on every split of
the row kernels; blocks of many tiles."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.helpers import assert_close_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,G,bs,T,N", [(128, 15, 64, 6700, 700), (128, 64, 30, 5900, 330), (64, 15, 30, 8300, 330),
                                        (64, 100, 64, 4000, 700), (128, 16, 900, 300, 2000)])
def test_long_lists(dev, D, G, bs, T, N):
    from omnimem_b200 import ops
    g = torch.Generator().manual_seed(T)
    M, H = 2 * G - 3, 2
    q, k, v, do = (torch.randn(1, n, H, D, generator=g).to(torch.float16) for n in (M, N, N, M))
    NB, MG = -(-N // bs), 2
    ids = torch.full((1, MG, H, T), -1, dtype=torch.int32)
    picks = min(NB, 9)
    at = torch.rand(1, MG, H, T, generator=g).argsort(-1)[..., :picks].sort(-1).values
    ids.scatter_(-1, at, torch.rand(1, MG, H, NB, generator=g).argsort(-1)[..., :picks].to(torch.int32))
    kv, scale = ops.DenseKV(k.to(dev), v.to(dev)), D ** -0.5
    d = ids.to(dev)
    out, lse = ops.sel_fwd(q.to(dev), kv, d, bs, 1, scale, False, G)
    grads = ops.sel_bwd(q.to(dev), kv, d, out, lse, do.to(dev), bs, 1, scale, False, G)
    short = ids.gather(-1, at)
    o_ref, l_ref = O.selection_fwd(q.float(), k.float(), v.float(), short, bs, 1, scale, False, G)
    want = O.selection_bwd(q.float(), k.float(), v.float(), short, o_ref, l_ref, do.float(), bs, 1, scale, False, G)
    assert_close_bf16(out, o_ref, "out", 2e-2, 2e-3)
    for name, a, b in zip(("dq", "dk", "dv"), grads, want):
        assert_close_bf16(a, b, name, 2e-2, 2e-3)
