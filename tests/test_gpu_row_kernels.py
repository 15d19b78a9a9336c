"""The row kernels (selection forward, dQ, dK/dV of every geometry outside the tcgen05 kernels) at the edges of their
tiles: blocks around 16 / 32 / 64 tokens, groups around 16 / 32 / 64 / 128 queries, ragged ends, lists split over
several warps, batches, page pools and address-strided inputs, against the CPU oracle."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.helpers import assert_close_bf16

pytestmark = pytest.mark.gpu

# B, M, N, H, D, T, block, group, causal, dtype
CASES = [
    (1, 75, 400, 2, 128, 4, 30, 15, False, torch.bfloat16),      # four warps per list
    (1, 1500, 900, 12, 128, 5, 30, 15, True, torch.bfloat16),    # one warp per list
    (1, 780, 900, 12, 64, 6, 24, 12, False, torch.float16),      # two warps per list at D = 64
    (2, 100, 310, 2, 128, 3, 31, 16, True, torch.bfloat16),      # blocks one short of a tile, batch: a copy per half
    (1, 66, 330, 3, 64, 3, 33, 17, False, torch.bfloat16),       # one over: tiles of 32 and 1 token, groups of 16 and 1
    (1, 130, 520, 2, 128, 2, 65, 65, True, torch.float16),       # five row warps of eight; tiles of 32, 32, 1
    (1, 256, 300, 2, 64, 3, 100, 128, False, torch.bfloat16),    # the largest group
    (1, 40, 64, 2, 128, 7, 1, 1, False, torch.bfloat16),         # the smallest of everything
    (3, 45, 160, 1, 64, 2, 16, 15, True, torch.float16),         # a single head
    (1, 90, 250, 2, 128, 3, 64, 32, False, torch.float16),       # a last block cut off in its second tile
    (1, 1300, 90, 1, 128, 3, 30, 10, False, torch.bfloat16),     # buckets longer than the kernel's tile list
]


def _inputs(case, dev, seed=3):
    B, M, N, H, D, T, bs, G, causal, dt = case
    g = torch.Generator().manual_seed(seed)
    q, k, v, do = (torch.randn(B, n, H, D, generator=g).to(dt) for n in (M, N, N, M))
    NB, MG = -(-N // bs), -(-M // G)
    ids = torch.rand(B, MG, H, NB, generator=g).argsort(-1)[..., :T].to(torch.int32)
    ids = torch.nn.functional.pad(ids, (0, T - ids.shape[-1]), value=-1)
    ids[:, 0, :, -1] = -1
    return q, k, v, do, ids.contiguous()


@pytest.mark.parametrize("case", CASES, ids=[f"bs{c[6]}_g{c[7]}_d{c[4]}_b{c[0]}" for c in CASES])
def test_tile_edges(dev, case):
    from omnimem_b200 import ops
    B, M, N, H, D, T, bs, G, causal, dt = case
    q, k, v, do, ids = _inputs(case, dev)
    chunk = max(G, M // 2) // 7 * 7 or G                       # causal limits inside blocks, not only between them
    scale = D ** -0.5
    kv = ops.DenseKV(k.to(dev), v.to(dev))
    out, lse = ops.sel_fwd(q.to(dev), kv, ids.to(dev), bs, chunk, scale, causal, G)
    dq, dk, dv = ops.sel_bwd(q.to(dev), kv, ids.to(dev), out, lse, do.to(dev), bs, chunk, scale, causal, G)
    o_ref, l_ref = O.selection_fwd(q.float(), k.float(), v.float(), ids, bs, chunk, scale, causal, G)
    grads = O.selection_bwd(q.float(), k.float(), v.float(), ids, o_ref, l_ref, do.float(), bs, chunk, scale, causal, G)
    fin = torch.isfinite(l_ref)
    assert torch.equal(torch.isfinite(lse.cpu()), fin)
    assert torch.allclose(lse.cpu()[fin], l_ref[fin], atol=2e-3, rtol=1e-4)
    # bf16 / fp16 operands, fp32 sums: the helper's 2e-2 / 2e-3; sums over s entries grow by at most their number,
    # which these buckets keep below that of the contract's workload except the last case (130 groups per block)
    grow = max(1.0, (M / G) * T * bs / N / 32)
    for name, got, want in (("out", out, o_ref), ("dq", dq, grads[0]), ("dk", dk, grads[1]), ("dv", dv, grads[2])):
        f = grow if name in ("dk", "dv") else 1.0
        assert_close_bf16(got, want, name, 2e-2 * f, 2e-3 * f)


def test_pages_and_strides(dev):
    """Pages of 30 tokens through the block table, and gradients from strided and expanded inputs, equal the dense ones."""
    from omnimem_b200 import ops
    case = (1, 90, 240, 3, 128, 4, 30, 15, False, torch.bfloat16)
    q, k, v, do, ids = (t.to(dev) for t in _inputs(case, dev))
    B, M, N, H, D, T, bs, G = case[:8]
    NB, scale = N // bs, D ** -0.5
    order = torch.randperm(H * NB, generator=torch.Generator().manual_seed(1)).to(dev)
    pool = lambda x: torch.empty(H * NB, bs, D, dtype=x.dtype, device=dev).index_copy_(
        0, order, x[0].view(NB, bs, H, D).permute(2, 0, 1, 3).reshape(H * NB, bs, D))
    paged = ops.PagedKV(pool(k), pool(v), order.view(H, NB).to(torch.int32), N, bs)
    dense = ops.DenseKV(k, v)
    out, lse = ops.sel_fwd(q, dense, ids, bs, 1, scale, False, G)
    out_p, lse_p = ops.sel_fwd(q, paged, ids, bs, 1, scale, False, G)
    assert torch.equal(out, out_p) and torch.equal(lse, lse_p)
    want = ops.sel_bwd(q, dense, ids, out, lse, do, bs, 1, scale, False, G)
    for got, w in zip(ops.sel_bwd(q, paged, ids, out, lse, do, bs, 1, scale, False, G), want):
        assert torch.equal(got, w)
    # one upstream row for all queries, as sum().backward() gives it: stride 0, which no tensor map describes
    row = do[:, :1].expand(B, M, H, D)
    want = ops.sel_bwd(q, dense, ids, out, lse, row.contiguous(), bs, 1, scale, False, G)
    for got, w in zip(ops.sel_bwd(q, dense, ids, out, lse, row, bs, 1, scale, False, G), want):
        assert torch.equal(got, w)


def test_values_outside_the_list_do_not_leak(dev):
    """A NaN in a token that no group lists stays out of every result (copies bring whole tiles)."""
    from omnimem_b200 import ops
    case = (1, 60, 300, 2, 128, 3, 30, 15, False, torch.bfloat16)
    q, k, v, do, _ = (t.to(dev) for t in _inputs(case, dev))
    ids = torch.tensor([0, 2, 8], dtype=torch.int32, device=dev).expand(1, 4, 2, 3).contiguous()
    k[:, 30:60], v[:, 30:60], k[:, 90:240], v[:, 90:240], k[:, 270:], v[:, 270:] = (float("nan"),) * 6
    kv = ops.DenseKV(k, v)
    out, lse = ops.sel_fwd(q, kv, ids, 30, 1, 128 ** -0.5, False, 15)
    grads = ops.sel_bwd(q, kv, ids, out, lse, do, 30, 1, 128 ** -0.5, False, 15)
    assert all(bool(torch.isfinite(t).all()) for t in (out, lse, *grads))


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_scales_that_are_not_positive(dev, scale):
    """Masked columns stay masked whatever the sign of the scale (ragged tiles, causal limits inside a block)."""
    from omnimem_b200 import ops
    case = (1, 90, 250, 2, 128, 3, 30, 15, True, torch.bfloat16)
    q, k, v, _, ids = _inputs(case, dev)
    out, lse = ops.sel_fwd(q.to(dev), ops.DenseKV(k.to(dev), v.to(dev)), ids.to(dev), 30, 35, scale, True, 15)
    o_ref, l_ref = O.selection_fwd(q.float(), k.float(), v.float(), ids, 30, 35, scale, True, 15)
    fin = torch.isfinite(l_ref)
    assert torch.equal(torch.isfinite(lse.cpu()), fin)
    assert torch.allclose(lse.cpu()[fin], l_ref[fin], atol=2e-3, rtol=1e-4)
    assert_close_bf16(out, o_ref, "out", 2e-2, 2e-3)
