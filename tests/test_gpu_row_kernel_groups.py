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
    # a result x is rounded to 16 bits (at most 2^-9 |x|) and sums products of factors that are (P or dS, 2^-9 each, of
    # either sign: some 2^-9 of the sum's own size): 2^-8 rms(x) on average and six times that at most, that is 4e-3 and 2.4e-2
    # per unit of rms(x); the contract's 2e-3 and 2e-2 for results smaller than that
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        f = max(1.0, 2 * b.float().square().mean().sqrt().item())
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


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("D,dt", [(128, torch.bfloat16), (64, torch.float16)])
@pytest.mark.parametrize("G", [7, 8, 16, 17, 32, 33, 48, 49, 64, 65, 128])
@pytest.mark.parametrize("bs", [1, 3, 4, 15, 16, 23, 24])
def test_short_blocks(dev, bs, G, D, dt, spread):
    """Around the sizes where packed tiles take over from a tile per block (a list of which several slots are empty)."""
    _case(dev, 1, 2 * G + 3, 9 * bs, 2, D, 12, bs, G, G % 2 == 1, dt, spread, G + bs)


@pytest.mark.parametrize("G", [64, 128])
def test_more_lists_than_fit_at_once(dev, G):
    """D = 64 with more warps than the chip holds: four warps share a ring."""
    _case(dev, 1, G * 101 + 7, 200, 24, 64, 1, 40, G, False, torch.bfloat16, False, 5)
