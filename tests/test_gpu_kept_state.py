"""Objects that the native host path keeps something of between calls: what their owner changes is seen by the next call."""
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
