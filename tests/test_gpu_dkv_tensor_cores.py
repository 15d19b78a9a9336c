"""dK / dV of blocks of at most 32 tokens on the tensor cores, at the edges of its tiles: groups of several 16-row pieces,
a 32nd token, single tokens and queries, buckets around a whole number of tiles, batches, both head dims and types."""
import pytest
import torch

import tests.test_gpu_row_kernels as rows

pytestmark = pytest.mark.gpu

# B, M, N, H, D, T, block, group, causal, dtype
CASES = [
    (1, 200, 320, 2, 128, 4, 32, 40, False, torch.bfloat16),     # three pieces per group, barriers behind the V tile
    (2, 256, 170, 2, 64, 3, 17, 128, True, torch.float16),       # eight pieces per group, a short last group
    (1, 64, 40, 1, 128, 1, 31, 16, False, torch.float16),        # exactly one tile
    (1, 80, 40, 1, 64, 1, 32, 16, False, torch.bfloat16),        # one piece more
    (2, 77, 63, 3, 128, 5, 8, 7, True, torch.bfloat16),
    (1, 33, 50, 2, 64, 9, 1, 33, False, torch.float16),          # one token per block, one row in the last piece
]


@pytest.mark.parametrize("case", CASES, ids=[f"bs{c[6]}_g{c[7]}_d{c[4]}_b{c[0]}" for c in CASES])
def test_tile_edges(dev, case):
    rows.test_tile_edges(dev, case)


def test_same_bits_every_time(dev):
    from omnimem_b200 import ops
    case = (1, 1500, 900, 4, 128, 8, 30, 15, True, torch.bfloat16)
    q, k, v, do, ids = (t.to(dev) for t in rows._inputs(case, dev))
    kv = ops.DenseKV(k, v)
    out, lse = ops.sel_fwd(q, kv, ids, 30, 150, 0.1, True, 15)
    first = ops.sel_bwd(q, kv, ids, out, lse, do, 30, 150, 0.1, True, 15)
    for _ in range(3):
        for a, b in zip(first, ops.sel_bwd(q, kv, ids, out, lse, do, 30, 150, 0.1, True, 15)):
            assert torch.equal(a, b)
