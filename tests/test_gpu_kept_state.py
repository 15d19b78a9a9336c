"""Objects that the native host path keeps something of between calls: what their owner changes is seen by the next call."""
import copy
import pickle

import pytest
import torch

pytestmark = pytest.mark.gpu


def _freqs(D=128, rows=64):
    from omnimem_b200.rollout import rope_table
    return torch.cat([rope_table(rows, D - 4 * (D // 6)), rope_table(rows, 2 * (D // 6)), rope_table(rows, 2 * (D // 6))], 1)


def _rand(dev, *shape, seed=0):
    g = torch.Generator(device=dev).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=dev).to(torch.bfloat16)


@pytest.mark.parametrize("change", [dict(start_frame=9), dict(grid_hw=(4, 2)), dict(grid_hw=[4, 2], pool=[1, 2, 1])])
def test_rope_geometry_may_change_after_the_first_use(dev, change):
    from omnimem_b200.cache import BlockKVCache, RopeSpec, rope_apply
    x = _rand(dev, 24, 2, 128)
    used, fresh = RopeSpec(_freqs(), (2, 4), 3), RopeSpec(_freqs(), (2, 4), 3)
    caches = [BlockKVCache(2, 128, 8, 4, device=dev, host_tier=False) for _ in range(2)]
    before = rope_apply(x, used)
    for rope, cache in ((used, caches[0]), (fresh, caches[1])):
        for name, value in change.items():
            setattr(rope, name, value)
        cache.append(x, x, rope=rope)
    assert torch.equal(rope_apply(x, used), rope_apply(x, fresh)) and not torch.equal(rope_apply(x, used), before)
    assert torch.equal(caches[0].k_pool, caches[1].k_pool)


def test_rope_refuses_another_head_dim_after_the_first_use(dev):
    from omnimem_b200.cache import RopeSpec, rope_apply
    rope = RopeSpec(_freqs(), (2, 4), 3)
    rope_apply(_rand(dev, 24, 2, 128), rope)
    with pytest.raises(RuntimeError, match="head dim 64"):
        rope_apply(_rand(dev, 24, 2, 64), rope)


def _model(dev):
    from omnimem_b200 import rollout as R
    shape = R.WanShape(dim=256, ffn_dim=512, num_heads=2, num_layers=2, text_dim=64, text_len=16)
    plan = R.RolloutPlan(latent_frames=6, latent_h=8, latent_w=16, topk=2, window_chunks=2, exclude_window_chunks=2)
    model, caches = R.build(shape, plan, dev, seed=1)
    latents, raw = _rand(dev, 1, shape.in_dim, 3, 8, 16), _rand(dev, 1, 16, 64)

    def forward(m=model, start=0):
        for c in caches:
            c.reset()
        with torch.no_grad():
            return m(latents, 500.0, m.text_embedding(raw), start, caches)
    return R, model, forward


def test_rotary_table_changed_in_place_between_forwards(dev):
    """However the model's table changes, the next forward is that of a model that never used another one."""
    R, model, forward = _model(dev)
    first = forward()
    assert torch.equal(forward(), first)
    changes = (lambda f: f.mul_(f), lambda f: f.data.mul_(f), lambda f: f.numpy().__imul__(f.numpy()), lambda f: f.copy_(f * f))
    for change in changes:
        model.freqs = torch.cat([R.rope_table(1024, 44), R.rope_table(1024, 42), R.rope_table(1024, 42)], dim=1)
        forward()
        change(model.freqs)
        got, model._rope = forward(), None
        assert torch.equal(got, forward()) and not torch.equal(got, first)
    model.freqs = model.freqs.to(dev)
    on_device = forward()
    model.freqs.data.mul_(model.freqs)
    got, model._rope = forward(), None
    assert torch.equal(got, forward()) and not torch.equal(got, on_device)


def test_rotary_tables_stay_on_their_stream(dev):
    """The copies are taken over by later specs on the stream they were made on; another stream makes its own."""
    from omnimem_b200.cache import RopeSpec, rope_apply
    x, freqs, side = _rand(dev, 24, 2, 128), _freqs(), torch.cuda.Stream()
    first = RopeSpec(freqs, (2, 4), 3)
    want = rope_apply(x, first)
    second = RopeSpec(freqs, (2, 4), 3, like=first)
    assert torch.equal(rope_apply(x, second), want) and second._tables is first._tables
    third = RopeSpec(freqs, (2, 4), 3, like=second)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = rope_apply(x, third)
    side.synchronize()
    assert torch.equal(got, want) and third._tables is not first._tables


def test_kv_sources_may_change_between_calls(dev):
    """The forward, the whole backward and its first half read the same fields, as they are at the call."""
    from omnimem_b200 import ops
    H, D, G, n = 2, 128, 64, 192
    q, k, v, k2, v2 = (_rand(dev, 1, n, H, D, seed=i) for i in range(5))
    ids = torch.arange(3, dtype=torch.int32, device=dev).expand(1, 3, H, 3).contiguous()

    def results(kv, backward=True):
        out, lse = ops.sel_fwd(q, kv, None if isinstance(kv, ops.PtrKV) else ids, 64, 1, 0.1, False, G)
        if not backward:
            return [out, lse]
        dq, delta = ops.sel_bwd_dq(q, kv, ids, out, lse, q, 64, 1, 0.1, False, G)
        return [out, lse, dq, delta, *ops.sel_bwd(q, kv, ids, out, lse, q, 64, 1, 0.1, False, G)]

    def same(a, b):
        return all(x.shape == y.shape and torch.equal(x, y) for x, y in zip(a, b, strict=True))

    kv = ops.DenseKV(k, v)
    first = results(kv)
    kv.n_tokens = 100                                                     # the rest of the tokens is not there
    assert same(results(kv), results(ops.DenseKV(k[:, :100], v[:, :100]))) and not same(results(kv)[:2], first[:2])
    kv.k, kv.v, kv.n_tokens = k2, v2, n
    assert same(results(kv), results(ops.DenseKV(k2, v2)))

    pools = [t.view(3, 64, H, D).permute(2, 0, 1, 3).reshape(3 * H, 64, D).contiguous() for t in (k[0], v[0], k2[0], v2[0])]
    table = torch.arange(3 * H, dtype=torch.int32, device=dev).view(H, 3)
    other = table.flip(0).contiguous()
    kv = ops.PagedKV(*pools[:2], table, n, 64)
    assert same(results(kv), first)
    kv.n_tokens = 100
    assert same(results(kv), results(ops.PagedKV(*pools[:2], table, 100, 64)))
    kv.n_tokens, kv.block_table = n, other
    assert same(results(kv), results(ops.PagedKV(*pools[:2], other, n, 64)))
    kv.k_pool, kv.v_pool, kv.block_table = pools[2], pools[3], table
    assert same(results(kv), results(ops.DenseKV(k2, v2)))

    def addresses(t):
        return t.data_ptr() + 2 * (ids.long() * 64 * H * D + torch.arange(H, device=dev).view(1, 1, H, 1) * D)

    kv = ops.PtrKV(addresses(k), addresses(v), H * D)
    ops.sel_fwd(q, kv, None, 64, 1, 0.1, False, G)
    kv.ptr_k, kv.ptr_v = addresses(k2), addresses(v2)
    assert same(results(kv, False), results(ops.PtrKV(addresses(k2), addresses(v2), H * D), False))
    kv.stride_bn = D                                                      # other rows of the same memory
    assert same(results(kv, False), results(ops.PtrKV(addresses(k2), addresses(v2), D), False))


def test_cache_tensors_may_be_replaced(dev):
    """Appends and touches write the tensors that the cache has now, as the page moves and the attention do."""
    from omnimem_b200.cache import BlockKVCache
    H, D = 2, 128
    k, v = _rand(dev, 200, H, D, seed=1), _rand(dev, 200, H, D, seed=2)
    ids = torch.arange(4, dtype=torch.int32, device=dev).expand(1, 1, H, 4).contiguous()
    kept, moved = (BlockKVCache(H, D, 8, 4, device=dev, host_tier=False) for _ in range(2))
    names = ("k_pool", "v_pool", "block_table", "page_owner", "page_stamp", "k_pooled", "v_pooled", "_stamp32", "status", "counters")
    for step in range(3):
        old = [getattr(moved, n) for n in names]
        for n, t in zip(names, old):
            setattr(moved, n, t.clone())
        before = [t.clone() for t in old]
        for cache in (kept, moved):
            cache.append(k[step * 60:step * 60 + 80], v[step * 60:step * 60 + 80], pos0=step * 60)
            cache.touch(ids)
        assert all(torch.equal(getattr(kept, n), getattr(moved, n)) for n in names)
        assert all(map(torch.equal, old, before))


COPIES = [copy.copy, copy.deepcopy, lambda x: pickle.loads(pickle.dumps(x))]


@pytest.mark.parametrize("duplicate", COPIES)
def test_used_objects_can_be_copied(dev, duplicate):
    from omnimem_b200 import ops
    from omnimem_b200.cache import RopeSpec, rope_apply
    x = _rand(dev, 1, 128, 2, 128)
    rope = RopeSpec(_freqs(), (4, 8), 3)
    want = rope_apply(x[0], rope)
    other = duplicate(rope)
    other.start_frame = 5
    assert torch.equal(rope_apply(x[0], duplicate(rope)), want) and not torch.equal(rope_apply(x[0], other), want)
    ids = torch.zeros(1, 2, 2, 1, dtype=torch.int32, device=dev)
    table = torch.arange(4, dtype=torch.int32, device=dev).view(2, 2)
    pool = _rand(dev, 4, 64, 128)
    for kv in (ops.DenseKV(x, x), ops.PagedKV(pool, pool, table, 128, 64)):
        want = ops.sel_fwd(x, kv, ids, 64, 1, 0.1, False, 64)
        assert all(map(torch.equal, ops.sel_fwd(x, duplicate(kv), ids, 64, 1, 0.1, False, 64), want))


@pytest.mark.parametrize("duplicate", COPIES[1:])
@pytest.mark.parametrize("host_tier", [False, True])
def test_used_caches_can_be_copied(dev, duplicate, host_tier):
    """The copy goes its own way, its host tier included, and meets what the original would have met."""
    from omnimem_b200.cache import BlockKVCache
    H, D = 2, 128
    cache = BlockKVCache(H, D, 12 if host_tier else 32, 16, device=dev, host_tier=host_tier, write_behind=False)
    for i in range(8):
        cache.append(_rand(dev, 64, H, D, seed=i), _rand(dev, 64, H, D, seed=100 + i))
    assert (cache.stats()["pages_evicted"] > 0) == host_tier
    other = duplicate(cache)
    q = _rand(dev, 1, 64, H, D, seed=9)
    ids = torch.tensor([0, 1, 6], dtype=torch.int32, device=dev).expand(1, 1, H, 3).contiguous()
    for i in range(2):
        outs = [c.selection_attention(q, ids) for c in (cache, other)]
        assert torch.equal(*outs) and cache.stats() == other.stats() and cache.n_tokens == other.n_tokens
        for c in (cache, other):
            c.append(_rand(dev, 64, H, D, seed=50 + i), _rand(dev, 64, H, D, seed=60 + i))
    other.append(q[0], q[0])
    assert other.n_tokens == cache.n_tokens + 64
    for c in (cache, other):
        c.check_status()


@pytest.mark.parametrize("duplicate", COPIES[1:])
def test_used_models_can_be_copied(dev, duplicate):
    R, model, forward = _model(dev)
    want = forward()
    other = duplicate(model)
    assert torch.equal(forward(other), want)
    with torch.no_grad():
        other.blocks[0].self_attn.q.weight.zero_()
    assert not torch.equal(forward(other), want) and torch.equal(forward(), want)
