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


def _setup(dev):
    R, shape, plan = _tiny()
    model, caches = R.build(shape, plan, dev, seed=1)
    g = torch.Generator(device=dev).manual_seed(2)
    rand = lambda *s: torch.randn(*s, generator=g, device=dev).to(torch.bfloat16)
    for p in model.parameters():                       # biases and norm weights that are not 0 and 1
        with torch.no_grad():
            p.add_(0.05 * torch.randn(p.shape, generator=g, device=dev))
    latents, raw = [rand(1, shape.in_dim, 3, 8, 16) for _ in range(2)], rand(1, 16, 64)

    def forward(eager=False):
        """Two chunks in a row; the layers take their eager form where gradients are on."""
        for c in caches:
            c.reset()
        with torch.set_grad_enabled(eager):
            context = model.text_embedding(raw)
            return torch.cat([model(x, 500.0, context, 3 * i, caches).detach() for i, x in enumerate(latents)])
    return model, forward


def _agree(got, want):
    # two bf16 blocks in a row, their activations rounded at other places: some four roundings of 2^-9 each
    assert (got.float() - want.float()).norm() <= 1e-2 * want.float().norm()


def test_the_fused_model_computes_what_its_eager_form_does(dev):
    model, forward = _setup(dev)
    assert all(b.fusable(torch.bfloat16) for b in model.blocks)
    _agree(forward(), forward(eager=True))


LAYERS = ("self_attn", "self_attn.q", "self_attn.k", "self_attn.v", "self_attn.g_proj", "self_attn.norm_q", "self_attn.norm_k",
          "self_attn.o", "norm3", "cross_attn", "cross_attn.q", "cross_attn.k", "cross_attn.v", "cross_attn.norm_q", "cross_attn.norm_k",
          "cross_attn.o", "ffn", "ffn.0", "ffn.1", "ffn.2", "")


@pytest.mark.parametrize("layer", LAYERS)
def test_a_layer_with_a_forward_of_its_own_is_called(dev, layer):
    model, forward = _setup(dev)
    plain = forward()
    m = model.blocks[1].get_submodule(layer)
    own, calls = m.forward, []

    def scaled(*args, **kw):
        calls.append(layer)
        return own(*args, **kw) * 0.5

    m.forward = scaled
    got = forward()
    assert len(calls) == 2 and not torch.equal(got, plain)
    _agree(got, forward(eager=True))
    del m.forward
    assert torch.equal(forward(), plain)


def test_global_hooks_and_patched_classes_are_met(dev):
    from torch.nn.modules.module import register_module_forward_hook
    model, forward = _setup(dev)
    plain, seen = forward(), set()
    handle = register_module_forward_hook(lambda m, args, out: seen.add(m))
    forward()
    handle.remove()
    assert {m for n, m in model.named_modules() if n.startswith("blocks.")} <= seen
    own = torch.nn.Linear.forward
    try:
        torch.nn.Linear.forward = lambda self, x: 0.5 * own(self, x)
        got = forward()
        _agree(got, forward(eager=True))
        assert not torch.equal(got, plain)
    finally:
        torch.nn.Linear.forward = own
    assert torch.equal(forward(), plain)


def _without(layer, name):
    def change(model):
        for b in model.blocks:
            b.get_submodule(layer).register_parameter(name, None)
    return pytest.param(change, id=f"{layer} without {name}")


def _replaced(layer, make, what):
    def change(model):
        for b in model.blocks:
            path, _, name = layer.rpartition(".")
            old = b.get_submodule(layer)
            new = make(old).to(device=next(model.parameters()).device, dtype=torch.bfloat16)
            setattr(b.get_submodule(path), name, new)
    return pytest.param(change, id=f"{layer}: {what}")


def _parameter(layer, name, make, what):
    def change(model):
        for b in model.blocks:
            m = b.get_submodule(layer)
            setattr(m, name, torch.nn.Parameter(make(getattr(m, name).data)))
    return pytest.param(change, id=f"{layer}.{name}: {what}")


def _spread(t):
    return torch.stack([t, t], -1)[..., 0]                        # not contiguous


def _shifted(t):
    return torch.cat([t.new_zeros(1), t.flatten()])[1:].view_as(t)  # not aligned to 16 bytes


def _no_bias(old):
    return torch.nn.Linear(old.in_features, old.out_features, bias=False)


def _no_affine(old):
    return torch.nn.LayerNorm(old.normalized_shape, eps=old.eps, elementwise_affine=False)


VARIANTS = [_without(l, "bias") for l in ("self_attn.q", "self_attn.g_proj", "self_attn.o", "cross_attn.k", "cross_attn.o", "ffn.0", "ffn.2",
                                          "norm3")]
VARIANTS += [_replaced(l, _no_bias, "no bias") for l in ("self_attn.k", "cross_attn.v", "ffn.0", "ffn.2")]
VARIANTS += [_replaced("norm3", _no_affine, "no affine")]
VARIANTS += [_parameter(l, "weight", f, f.__name__) for l in ("self_attn.norm_q", "self_attn.norm_k", "cross_attn.norm_k", "norm3", "self_attn.v")
             for f in (_spread, _shifted)]
VARIANTS += [_parameter("", "modulation", f, f.__name__) for f in (_spread, _shifted)]
VARIANTS += [_parameter("self_attn.norm_q", "weight", torch.Tensor.float, "fp32")]


@pytest.mark.parametrize("moved", [False, True])
@pytest.mark.parametrize("change", VARIANTS)
def test_ordinary_variants_of_the_layers(dev, change, moved):
    """Layers without a bias, norms without a weight, parameters that lie otherwise: the eager form's result, also after
    the model has been moved (where the weights of the projections are laid together)."""
    model, forward = _setup(dev)
    plain = forward()
    change(model)
    if moved:
        model.to(dtype=torch.float32).to(dtype=torch.bfloat16)
    got = forward()
    _agree(got, forward(eager=True))
    assert got.shape == plain.shape and torch.isfinite(got.float()).all()


def test_moved_models_keep_types_and_ties(dev):
    """Laying weights together changes neither a parameter's type nor which layers share one."""
    model, forward = _setup(dev)
    attn, cross = model.blocks[0].self_attn, model.blocks[0].cross_attn
    attn.q.bias = torch.nn.Parameter(attn.q.bias.data.float())
    cross.k.weight = cross.v.weight
    model.to(dev)
    assert attn.q.bias.dtype == torch.float32 and attn.k.bias.dtype == torch.bfloat16 and attn.q.weight.dtype == torch.bfloat16
    assert cross.k.weight is cross.v.weight and cross.k.weight.data_ptr() == cross.v.weight.data_ptr()


@pytest.mark.parametrize("layer", ["self_attn.norm_q", "self_attn.norm_k", "cross_attn.norm_k", "norm3"])
def test_each_norm_has_an_eps_of_its_own(dev, layer):
    model, forward = _setup(dev)
    plain = forward()
    for b in model.blocks:
        b.get_submodule(layer).eps = 4.0
    got = forward()
    _agree(got, forward(eager=True))
    assert not torch.equal(got, plain)


class _Wrapped(torch.nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, *args, **kw):
        return self.inner(*args, **kw)


def _layer_norm(old):
    return torch.nn.LayerNorm(old.weight.numel())


def _rms_norm(old):
    from omnimem_b200.rollout import RMSNorm
    return RMSNorm(old.weight.numel(), old.eps)


KINDS = [_replaced(l, _layer_norm, "layer norm") for l in ("self_attn.norm_q", "self_attn.norm_k", "cross_attn.norm_q", "cross_attn.norm_k")]
KINDS += [_replaced("norm3", _rms_norm, "rms norm")]
KINDS += [_replaced(l, _Wrapped, "wrapped") for l in ("ffn", "ffn.0", "ffn.1", "self_attn", "cross_attn", "self_attn.q", "self_attn.o", "norm3")]
KINDS += [_replaced("ffn.1", lambda old: torch.nn.GELU(), "exact gelu"),
          _replaced("ffn", lambda old: torch.nn.Sequential(*old, torch.nn.Identity()), "longer")]


@pytest.mark.parametrize("change", KINDS)
def test_layers_of_another_kind(dev, change):
    """What a user puts in a layer's place is what runs there, also where it is one of the kinds that the fused form knows."""
    model, forward = _setup(dev)
    change(model)
    _agree(forward(), forward(eager=True))


def test_blocks_of_another_kind(dev):
    model, forward = _setup(dev)
    plain = forward(eager=True)
    model.blocks[1] = _Wrapped(model.blocks[1])
    _agree(forward(), plain)
