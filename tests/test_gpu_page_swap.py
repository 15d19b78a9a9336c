"""Evict and fetch in one kernel against an evict followed by a fetch: pages, host slots, tables and counters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page_bytes,n,owned", [(16, 1, 1), (16384, 37, 30), (16400, 5, 0), (40960, 12, 12), (4096 + 16, 9, 5)])
def test_swap_is_evict_then_fetch(dev, page_bytes, n, owned):
    from omnimem_b200 import _lib
    g = torch.Generator().manual_seed(n)
    pages_total, keys_total = n + 5, 4 * n + 8
    pool = torch.randint(0, 256, (2, pages_total, page_bytes), generator=g, dtype=torch.uint8)
    host = torch.randint(0, 256, (2, keys_total, page_bytes), generator=g, dtype=torch.uint8)
    pages = torch.randperm(pages_total, generator=g)[:n + 1].to(torch.int32)
    pages[n] = -1                                                       # no victim was found for the last miss
    keys = torch.randperm(keys_total, generator=g).to(torch.int32)
    owner = torch.full((pages_total,), -1, dtype=torch.int32)
    table = torch.full((keys_total,), -1, dtype=torch.int32)
    owner[pages[:owned].long()] = keys[:owned]
    table[keys[:owned].long()] = pages[:owned]
    fetch = torch.cat([torch.tensor([n + 1], dtype=torch.int32), keys[owned:owned + n + 1]])
    got = []
    for directions in ((0, 1), (4,)):
        d = [t.clone().to(dev) for t in (pool, owner, table, torch.zeros(pages_total, dtype=torch.int64),
                                         torch.zeros(4, dtype=torch.int64), pages, fetch)]
        p, o, t, stamp, counters, pg, ks = d
        h = host.clone().pin_memory()
        for direction in directions:
            _lib.call("nsa_cache_move_pages", direction, pg.data_ptr(), ks.data_ptr(), 0, ks.data_ptr(), n + 3, p[0].data_ptr(),
                      p[1].data_ptr(), page_bytes, h[0].data_ptr(), h[1].data_ptr(), t.data_ptr(), o.data_ptr(),
                      stamp.data_ptr(), 7, counters.data_ptr(), torch.cuda.current_stream(dev).cuda_stream)
        torch.cuda.synchronize()
        got.append([x.cpu() for x in (p, o, t, stamp, counters)] + [h.clone()])
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert got[1][4].tolist()[2:] == [owned, n]
