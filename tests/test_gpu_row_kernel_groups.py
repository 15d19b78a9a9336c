"""The row kernels over the group sizes at which their dispatch changes, against the CPU oracle: query rows per step of
dK/dV, thread blocks per group and tile heights of the forward and dQ; described by tensor maps and not."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.helpers import assert_close_bf16

pytestmark = pytest.mark.gpu


def _case(dev, B, M, N, H, D, T, bs, G, causal, dt, spread, seed):
    """`spread`: K, V and dO repeat one head (a stride of zero, which no tensor map describes)."""
    from omnimem_b200 import ops
    g = torch.Generator().manual_seed(seed)
    q, k, v, do = (torch.randn(B, n, 1 if spread and i else H, D, generator=g).to(dt).expand(B, n, H, D) for i, n in enumerate((M, N, N, M)))
    NB, MG = -(-N // bs), -(-M // G)
    ids = torch.rand(B, MG, H, NB, generator=g).argsort(-1)[..., :T].to(torch.int32)
    ids = torch.nn.functional.pad(ids, (0, T - ids.shape[-1]), value=-1).contiguous()
    chunk, scale = max(G, M // 2), D ** -0.5
    one = lambda t: t[:, :, :1].to(dev).expand(t.shape) if spread and t is not q else t.to(dev)
    kv = ops.DenseKV(one(k), one(v))
    out, lse = ops.sel_fwd(q.to(dev), kv, ids.to(dev), bs, chunk, scale, causal, G)
    got = (out, *ops.sel_bwd(q.to(dev), kv, ids.to(dev), out, lse, one(do), bs, chunk, scale, causal, G))
    o_ref, l_ref = O.selection_fwd(q.float(), k.float(), v.float(), ids, bs, chunk, scale, causal, G)
    want = (o_ref, *O.selection_bwd(q.float(), k.float(), v.float(), ids, o_ref, l_ref, do.float(), bs, chunk, scale, causal, G))
    fin = torch.isfinite(l_ref)
    assert torch.equal(torch.isfinite(lse.cpu()), fin)
    assert torch.allclose(lse.cpu()[fin], l_ref[fin], atol=2e-3, rtol=1e-4)
    # dK / dV sum over the M / G * T * bs / N groups that list a block: the contract's limits hold for up to 32 rows of them
    grow = max(1.0, (M / G) * T * bs / N / 32)
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        f = grow if name[1] in "kv" else 1.0
        assert_close_bf16(a, b, f"{bs}/{G} D{D} {name}", 2e-2 * f, 2e-3 * f)


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("D,dt", [(128, torch.float16), (64, torch.bfloat16)])
@pytest.mark.parametrize("G", [17, 32, 33, 48, 49, 63, 64, 65, 96, 97, 112, 128])
@pytest.mark.parametrize("bs", [33, 64, 100])
def test_larger_groups(dev, bs, G, D, dt, spread):
    # the last group is cut off inside its first tile, the last block inside its last one
    _case(dev, 1, 3 * G + 5, 5 * bs - 3, 2, D, 3, bs, G, G % 2 == 0, dt, spread, G)


@pytest.mark.parametrize("D,dt", [(128, torch.bfloat16), (64, torch.float16)])
@pytest.mark.parametrize("B,H", [(2, 3), (1, 1)])
def test_long_buckets_of_larger_groups(dev, B, H, D, dt):
    _case(dev, B, 64 * 70 + 9, 130, H, D, 2, 65, 64, False, dt, False, 1)        # more tiles than a bucket's list holds
