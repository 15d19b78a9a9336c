"""Selection of rows longer than 1024 blocks, the causal skip of the scoring kernel, and the inverted index of long and
short buckets, against sorts on the CPU."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(scores, visible, topk):
    """scores [.., NC] float64, visible the same: ids by (score descending, id ascending), -1 where nothing is visible."""
    order = torch.sort(torch.where(visible, scores, -float("inf")), dim=-1, descending=True, stable=True).indices[..., :topk]
    return torch.where(visible.gather(-1, order), order, -1)


# rows, columns, head dim, top-k, score pattern, causal, dtype
CASES = [
    (9, 1025, 64, 1, "random", False, torch.bfloat16),
    (9, 1092, 128, 16, "ties", True, torch.bfloat16),
    (700, 1090, 64, 16, "random", True, torch.float16),      # one warp per row
    (5, 1601, 64, 17, "few lanes", False, torch.bfloat16),   # two warps, one round per winner
    (3, 4099, 64, 64, "random", False, torch.bfloat16),
    (3, 9001, 64, 128, "ties", True, torch.bfloat16),        # eight warps
    (6, 2048, 64, 16, "few lanes", True, torch.float32),
    (40, 1100, 64, 33, "falling", True, torch.float32),
    (25, 98, 128, 16, "random", False, torch.float32),       # one row per thread
    (300, 1100, 64, 8, "ties", False, torch.float32),        # eight rows per thread, row steps dealt out
]


@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}x{c[1]}_t{c[3]}_{c[4].replace(' ', '')}" for c in CASES])
def test_long_rows(dev, case):
    from omnimem_b200 import ops
    MG, NC, D, T, pattern, causal, dtype = case
    H, g = 2, torch.Generator().manual_seed(NC)
    q, k = torch.zeros(1, MG, H, D), torch.zeros(1, NC, H, D)
    # small integers: every product and sum is exact, so the order is known to the last bit
    if pattern == "falling":
        n = torch.arange(NC - 1, -1, -1)
        k[..., 0], k[..., 1] = (n // 64).view(1, NC, 1), (n % 64).view(1, NC, 1)
        q[..., 0], q[..., 1] = 64, 1
    else:
        top = 2 if pattern == "ties" else 40
        k[..., :4] = torch.randint(-top, top, (1, NC, H, 4), generator=g).float()
        q[..., :4] = torch.randint(-3, 4, (1, MG, H, 4), generator=g).float()
        if pattern == "few lanes":
            q[..., 4], k[..., 4] = 16, torch.where(torch.arange(NC) % 256 < 10, 64.0, 0.0).view(1, NC, 1)
    block, chunk_k = 4, 100
    chunk = 3
    idx = ops.topk(q.to(dtype).to(dev), k.to(dtype).to(dev), T, 1.0, block, chunk, chunk_k, causal, q_group_size=2)
    scores = torch.einsum("bghd,bchd->bghc", q.double(), k.double())
    cols = torch.arange(NC)
    visible = torch.ones_like(scores, dtype=torch.bool)
    if causal:
        rows = torch.arange(MG) * 2 // chunk
        visible &= (cols * block // chunk_k).view(1, 1, 1, NC) <= rows.view(1, MG, 1, 1)
    assert torch.equal(idx.cpu().long(), _expected(scores, visible, T))


@pytest.mark.parametrize("MG,T,NS,causal,slots", [(50, 16, 40, True, False), (2000, 4, 30, False, True), (300, 8, 7, True, True),
                                                  (9000, 8, 50, False, False), (40000, 2, 3, False, True), (4000, 16, 9000, True, False)])
def test_inverted_index(dev, MG, T, NS, causal, slots):
    """Buckets from empty to all groups, staged in shared memory and not, in (group, slot) order."""
    from omnimem_b200 import _lib
    B, H, bs, G = 1, 2, 30, 15
    chunk = bs * max(1, NS // 3)
    ids = torch.randint(-1, NS + 1, (B, MG, H, T), generator=torch.Generator().manual_seed(MG), dtype=torch.int32)
    ids[:, :, :, 0] = 0                                            # one block that every group lists
    d = ids.to(dev)
    pairs = B * H * MG * T
    groups, slot, offsets = (torch.full((n,), -5, dtype=torch.int32, device=dev) for n in (pairs, pairs, B * H * (NS + 1)))
    lib = _lib.load()
    n = lib.nsa_inverted_index_workspace_bytes(B, H, NS)
    ws = torch.empty(max(n, 1), dtype=torch.uint8, device=dev)
    strides = (C.c_int64 * 4)(*d.stride())
    _lib.call("nsa_inverted_index_slots", d.data_ptr(), strides, B, MG, H, T, NS, bs, chunk, int(causal), G, groups.data_ptr(),
              offsets.data_ptr(), slot.data_ptr() if slots else None, ws.data_ptr(), n, torch.cuda.current_stream(dev).cuda_stream)
    g_of, t_of = torch.meshgrid(torch.arange(MG), torch.arange(T), indexing="ij")
    for h in range(H):
        i = ids[0, :, h].long()
        ok = (i >= 0) & (i < NS)
        if causal:
            ok &= i * bs // chunk <= g_of * G // chunk
        key = (i[ok] * MG + g_of[ok]) * T + t_of[ok]
        order = key.sort().indices
        count = torch.bincount(i[ok], minlength=NS)
        want = torch.cat([torch.zeros(1, dtype=torch.long), count.cumsum(0)])
        assert torch.equal(offsets.cpu().view(H, NS + 1)[h].long(), want)
        assert torch.equal(groups.cpu().view(H, -1)[h, :len(order)].long(), g_of[ok][order])
        if slots:
            assert torch.equal(slot.cpu().view(H, -1)[h, :len(order)].long(), t_of[ok][order])


@pytest.mark.parametrize("case", [
    (3, 8192, 64, 16, "random", False, torch.bfloat16),      # eight segments: still a thread block per row
    (3, 8193, 64, 16, "ties", True, torch.bfloat16),         # segments, the last one of one column
    (74, 9001, 64, 16, "random", True, torch.float16),       # the most rows that are split
    (75, 9001, 64, 16, "ties", False, torch.bfloat16),       # one more
    (1, 20000, 64, 1, "random", False, torch.bfloat16),
    (2, 17500, 64, 8, "few lanes", True, torch.float32),
    (3, 33000, 64, 17, "few lanes", False, torch.bfloat16),  # 32 warps per row
    (20, 17000, 64, 128, "ties", True, torch.bfloat16),      # 16
    (17, 1000, 64, 8, "random", True, torch.bfloat16),       # scores of 17 rows: warps with none
], ids=lambda c: f"{c[0]}x{c[1]}_t{c[3]}")
def test_few_long_rows(dev, case):
    test_long_rows(dev, case)
