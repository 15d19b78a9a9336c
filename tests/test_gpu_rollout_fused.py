"""The fused form of the rollout's layers: what it serves, what it refuses, and what it leaves to the eager form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tiny(frames=6, layers=2):
    from omnimem_b200 import rollout as R
    shape = R.WanShape(dim=256, ffn_dim=512, num_heads=2, num_layers=layers, text_dim=64, text_len=16)
    plan = R.RolloutPlan(latent_frames=frames, latent_h=8, latent_w=16, topk=2, window_chunks=2, exclude_window_chunks=2,
                         timesteps=(1000.0, 500.0))
    return R, shape, plan


def test_batches_are_refused(dev):
    """The caches hold one batch element: a batch of two raises, in the layer and in the model, and writes no cache."""
    R, shape, plan = _tiny()
    model, caches = R.build(shape, plan, dev, seed=1)
    x = torch.randn(2, 96, shape.dim, device=dev).to(torch.bfloat16)
    rope = R.RopeSpec(model.freqs, (4, 8), 0)
    with torch.no_grad():
        with pytest.raises(RuntimeError, match="batch size 1"):
            model.blocks[0].self_attn(x, caches[0], rope, 0)
        context = model.text_embedding(torch.randn(1, 16, 64, device=dev).to(torch.bfloat16))
        with pytest.raises(RuntimeError, match="batch size 1"):
            model(torch.randn(2, shape.in_dim, 3, 8, 16, device=dev).to(torch.bfloat16), 500.0, context, 0, caches)
    assert caches[0].n_tokens == 0 and caches[1].n_tokens == 0
