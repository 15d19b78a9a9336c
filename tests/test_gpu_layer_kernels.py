"""Row-wise kernels of a transformer layer (residual + norm + modulation, RMS norm, query / key norm + rotary embedding)
against the eager expressions they replace, at rows of every built length."""
import pytest
import torch
import torch.nn.functional as F

from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu

# bf16 / fp16 results of fp32 arithmetic in another order: one unit in the last place of the largest terms
ULP = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}


def _close(got, want, dtype, terms=4.0):
    tol = ULP[dtype] * terms
    assert (got.float() - want.float()).abs().max() <= tol * max(1.0, want.float().abs().max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,d", [(1, 8), (7, 248), (9, 256), (33, 520), (16, 1536), (5, 2048)])
def test_residual_norm(dev, rows, d, dtype):
    from omnimem_b200._lib import host
    g = torch.Generator(device=dev).manual_seed(rows + d)
    rand = lambda *s: torch.randn(*s, generator=g, device=dev)
    x, y = rand(1, rows, d).to(dtype), rand(1, rows, d).to(dtype)
    m, e = rand(3, d).to(dtype), rand(3, d)
    eps, none = 1e-6, (None, None)
    ln = lambda t: F.layer_norm(t.float(), (d,), eps=eps)
    vec = lambda i: m[i].float() + e[i]
    # no residual, modulated
    got_x, got = host.residual_norm(x, None, none, (m[0], e[0]), (m[1], e[1]), True, True, eps)
    assert torch.equal(got_x, x)
    _close(got, (ln(x) * (1 + vec(0)) + vec(1)).to(dtype), dtype)
    # gated residual, affine norm
    x2 = x + (y.float() * vec(2)).to(dtype)
    got_x, got = host.residual_norm(x, y, (m[2], e[2]), (m[0], None), (m[1], None), False, True, eps)
    assert torch.equal(got_x, x2)
    _close(got, F.layer_norm(x2, (d,), m[0], m[1], eps), dtype)
    # plain residual without a norm
    got_x, got = host.residual_norm(x, y, none, none, none, True, False, eps)
    assert torch.equal(got_x, x + y) and got is None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,D,grid", [(2, 128, (3, 5)), (4, 64, (4, 4)), (12, 128, (6, 7)), (8, 256, (1, 3))])
def test_qk_norm_rope(dev, H, D, grid, dtype):
    """Equal to the eager norm and the float64 rotary embedding up to the norm's last bit, keys in place."""
    from omnimem_b200._lib import host
    from omnimem_b200.cache import RopeSpec
    from omnimem_b200.rollout import rope_table
    d, frames, S = H * D, 2, 2 * grid[0] * grid[1]
    g = torch.Generator(device=dev).manual_seed(d)
    buf = torch.randn(S, 2 * d + 64, generator=g, device=dev).to(dtype)
    qw, kw = (1 + 0.1 * torch.randn(2, d, generator=g, device=dev)).to(dtype).unbind(0)
    freqs = torch.cat([rope_table(64, D - 4 * (D // 6)), rope_table(64, 2 * (D // 6)), rope_table(64, 2 * (D // 6))], 1)
    rope = RopeSpec(freqs, grid, 3)
    q, k = buf[:, :d], buf[:, d:2 * d]
    rms = lambda t, w: F.rms_norm(t.float(), (d,), w.float(), 1e-6).to(dtype)
    want = [O.reorder_rope_apply(rms(t, w).view(S, H, D).cpu(), (frames, *grid), freqs, 3, (1, 1, 1)) for t, w in ((q, qw), (k, kw))]
    tail = buf[:, 2 * d:].clone()
    got_q = host.qk_norm_rope(q, k, qw, kw, 1e-6, H, rope.native(dev, D))
    _close(got_q.cpu(), want[0], dtype)
    _close(k.reshape(S, H, D).cpu(), want[1], dtype)
    assert torch.equal(buf[:, 2 * d:], tail)
    _close(host.rms_rows(buf[:, :d], qw, 1e-6), rms(buf[:, :d], qw), dtype)


def test_touch_without_lists_stamps_and_counts_like_the_lists(dev):
    from omnimem_b200.cache import BlockKVCache
    H, D, MB = 3, 128, 40
    g = torch.Generator().manual_seed(2)
    caches = [BlockKVCache(H, D, H * MB, MB, device=dev, host_tier=False) for _ in range(2)]
    kv = torch.randn(20 * 64, H, D, generator=g).to(torch.bfloat16).to(dev)
    ids = torch.randint(-1, 30, (1, 7, H, 5), generator=g, dtype=torch.int32).to(dev)       # some without a page, some -1
    for c in caches:
        c.append(kv, kv)
    caches[0].touch(ids)
    caches[1].touch(ids, return_lists=True)
    assert torch.equal(caches[0].counters, caches[1].counters) and torch.equal(caches[0].page_stamp, caches[1].page_stamp)
    assert caches[0].stats()["misses"] > 0 and caches[0].stats()["hits"] > 0


def test_packed_projections_follow_their_layers(dev):
    """One product over layers whose weights lie together sees every way in which a parameter or a layer can change."""
    from omnimem_b200.rollout import CrossAttention, WanShape, _plain
    m = CrossAttention(WanShape(dim=256, num_heads=2)).to(device=dev, dtype=torch.bfloat16)
    x = torch.randn(5, 256, device=dev).to(torch.bfloat16)

    def same():
        for got, layer in zip(m.project(x), (m.k, m.v)):
            want = layer(x)
            assert got.shape == want.shape and (got.float() - want.float()).abs().max() <= 2 ** -6 * want.float().abs().max()

    state = {n: t.clone() for n, t in m.state_dict().items()}
    fresh = lambda: torch.nn.Parameter(torch.randn_like(m.v.bias))
    with torch.no_grad():
        assert m._joined((m.k, m.v)) is not None and m.k.weight.untyped_storage().data_ptr() == m.v.weight.untyped_storage().data_ptr()
        changes = (lambda: m.k.weight.mul_(2), lambda: m.k.weight.data.copy_(torch.randn_like(m.k.weight)),
                   lambda: m.load_state_dict(state), lambda: setattr(m.v, "bias", fresh()),
                   lambda: m.to(dtype=torch.float32).to(dtype=torch.bfloat16), lambda: setattr(m.v, "bias", fresh()),
                   lambda: setattr(m.v.weight, "data", torch.randn_like(m.v.weight)),
                   lambda: m.load_state_dict(state, assign=True))
        same()
        for change in changes:
            change()
            same()
    assert _plain(torch.bfloat16, m.k, m.v) and not _plain(torch.float16, m.k)
    m.k.register_forward_hook(lambda *a: None)
    assert not _plain(torch.bfloat16, m.k)
    m.v = torch.nn.Sequential(m.v)
    assert not _plain(torch.bfloat16, m.v)


@pytest.mark.parametrize("H,D", [(2, 128), (4, 64)])
def test_rotary_tables_built_on_the_device(dev, H, D):
    """The copies that split a table on the device are the launches directly in front of the kernel that reads them: the
    results are those of a table that was complete long before."""
    from omnimem_b200._lib import host
    from omnimem_b200.cache import RopeSpec
    from omnimem_b200.rollout import rope_table
    d, S = H * D, 2 * 3 * 5
    g = torch.Generator(device=dev).manual_seed(D)
    freqs = torch.cat([rope_table(64, D - 4 * (D // 6)), rope_table(64, 2 * (D // 6)), rope_table(64, 2 * (D // 6))], 1)
    w = torch.ones(d, device=dev, dtype=torch.bfloat16)
    for start in range(8):
        q, k = torch.randn(2, S, d, generator=g, device=dev).to(torch.bfloat16).unbind(0)
        got = []
        for table in (freqs, freqs.to(dev)):
            kk = k.clone()
            rope = RopeSpec(table, (3, 5), start)
            got.append((host.qk_norm_rope(q, kk, w, w, 1e-6, H, rope.native(dev, D)), kk))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
