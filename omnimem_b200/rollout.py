"""Causal chunk-by-chunk rollout of a Wan2.1-T2V-1.3B-shaped transformer whose self-attention is the
three-branch native sparse attention, driven through this library's block cache and kernels.

This is the CALLER of the selection path, re-typed from the shapes of the reference so that the
path can be measured where it is used: 30 blocks, width 1536, 12 heads of 128, feed-forward 8960,
patch 1x2x2 over 16 latent channels, 512 x 4096 text conditioning, random bf16 weights, synthetic
inputs.  Per chunk of three latent frames (4680 tokens) it runs four denoising forwards and one
cache-write forward at t = 0 (pipelines/pipeline_wan_causal.py:349-495); a layer does what
CausalNSSelfAttention.forward does in its rollout branch (models/transformers/
causal_wan_nsa_model.py:354-553): projections and gates, rotary embedding with the frame offset,
cache update with pooled keys / values, compressed attention over the pooled history, sliding-window
attention over the last chunks, top-k block selection and selection attention over the paged
history, gated sum, output projection.

What runs where:
  * linear layers (the feed-forward's GELU in its epilogue), cross-attention (SDPA), embeddings: torch;
  * residual add + layer norm + modulation (one kernel per stop of the residual stream), query / key norm +
    rotary embedding (one kernel), pooling + page append (one kernel), query-group pooling, scoring + top-k,
    LRU touch / evict / fetch, all THREE attention branches (the selection forward kernel over the selected
    pages; the range forward kernel over the window's pages and over the pooled history as a dense tensor),
    and the gated sum: this library.
The fused form serves 16-bit activations without gradients, which is what a rollout is; anything else takes the
eager form of the same layer.
Tokens stay in (frame, row, column) order and a block is 64 consecutive tokens (the reference pools
spatial tiles of 15 x 2 tokens; 64-token blocks cut across rows and chunk boundaries, which the block
cache is built for).  The window starts at the block that holds its first token.
"""
from __future__ import annotations

import math
import time
from dataclasses import dataclass, field
from typing import List, Optional

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.nn.modules.module import _has_any_global_hook

from . import ops
from ._lib import NSABackendError, host
from .cache import BlockKVCache, RopeSpec, rope_apply
from .nsa.ops.index_topk import should_use_selection_attention


@dataclass
class WanShape:
    dim: int = 1536
    ffn_dim: int = 8960
    num_heads: int = 12
    num_layers: int = 30
    in_dim: int = 16
    out_dim: int = 16
    patch: tuple = (1, 2, 2)
    text_dim: int = 4096
    text_len: int = 512
    freq_dim: int = 256
    eps: float = 1e-6


@dataclass
class RolloutPlan:
    latent_frames: int = 21
    frames_per_chunk: int = 3
    latent_h: int = 60                      # 480 / 8
    latent_w: int = 104                     # 832 / 8
    timesteps: tuple = (1000.0, 750.0, 500.0, 250.0)
    topk: int = 16
    block: int = 64
    group: int = 64
    window_chunks: int = 3                  # sliding window of the swa branch, in chunks (the current one included)
    exclude_window_chunks: int = 3          # the selection skips what the window covers ...
    progressive_exclude: bool = True        # ... once the history is longer than the window
    cache_cap_frames: Optional[int] = None  # resident full-resolution K/V per layer, in latent frames (None: everything)
    new_prompt_every: Optional[int] = None  # a fresh conditioning tensor every this many latent frames
    seed: int = 0


class SectionTimer:
    """CUDA-event brackets per named section of a layer, summed over layers and forwards - the role
    of the reference's TripleAttnProfiler (utils/attn_profiler.py:10-133: cache, cmp, swa, slc_topk,
    slc_attn).  Off by default: the brackets cost launches of their own."""

    def __init__(self):
        self.events = {}

    class _Span:
        def __init__(self, owner, name):
            self.owner, self.name = owner, name

        def __enter__(self):
            self.a = torch.cuda.Event(enable_timing=True)
            self.b = torch.cuda.Event(enable_timing=True)
            self.a.record()

        def __exit__(self, *exc):
            self.b.record()
            self.owner.events.setdefault(self.name, []).append((self.a, self.b))

    def __call__(self, name):
        return SectionTimer._Span(self, name)

    def summary_ms(self, per: int = 1) -> dict:
        """Total milliseconds per section divided by `per` (e.g. the number of forwards)."""
        torch.cuda.synchronize()
        return {k: round(sum(a.elapsed_time(b) for a, b in v) / per, 3) for k, v in self.events.items()}


class _NoTimer:
    def __call__(self, name):
        return self

    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_NO_TIMER = _NoTimer()


def rope_table(max_len: int, dim: int, theta: float = 10000.0) -> torch.Tensor:
    """complex128 [max_len, dim/2] (rope_params, wan_model.py:37-43)."""
    ang = torch.outer(torch.arange(max_len, dtype=torch.float64),
                      1.0 / torch.pow(theta, torch.arange(0, dim, 2, dtype=torch.float64) / dim))
    return torch.polar(torch.ones_like(ang), ang)


def sinusoidal_embedding(dim: int, t: torch.Tensor) -> torch.Tensor:
    half = dim // 2
    pos = t.to(torch.float64)
    freq = torch.pow(10000.0, -torch.arange(half, dtype=torch.float64, device=t.device) / half)
    x = torch.outer(pos, freq)
    return torch.cat([x.cos(), x.sin()], dim=1).float()


class RMSNorm(nn.Module):
    def __init__(self, dim, eps):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(dim))
        self.eps = eps

    def forward(self, x):
        return F.rms_norm(x.float(), (x.shape[-1],), self.weight.float(), self.eps).to(x.dtype)


def _fused(x: torch.Tensor) -> bool:
    """Whether the fused kernels serve activations x [.., d] (layer.cu): 16-bit, no gradients, no autocast, rows they are
    built for, and no hook that every module's call has to run."""
    return x.is_cuda and x.dtype in (torch.bfloat16, torch.float16) and not torch.is_grad_enabled() \
        and not torch.is_autocast_enabled("cuda") and x.shape[-1] in (256, 512, 1024, 1536, 2048) \
        and not _has_any_global_hook()


def _row(p, dtype: torch.dtype) -> bool:
    """Whether the row kernels can read vector (or rows of vectors) p as it lies."""
    return type(p) in (nn.Parameter, torch.Tensor) and p.dtype == dtype and p.is_contiguous() and p.data_ptr() % 16 == 0


def _are(kinds: tuple, dtype: torch.dtype, mods: tuple) -> bool:
    """Whether the fused form may use the parameters of `mods` without calling them: modules exactly of these kinds (not
    something a user put in their place), whose call does nothing but what their class does as it is written here (no hooks,
    no `forward` of their own: offloading and adapter libraries set one; none put on the class; not compiled), with
    parameters of the activations' type.  A linear layer may lack its bias, a norm has to have all that it is built with."""
    return host.plain(mods, kinds, _PLAIN, nn.Parameter, dtype)


def _plain(dtype: torch.dtype, *mods: nn.Module) -> bool:
    kinds = tuple(map(type, mods))
    return all(k in (nn.Linear, nn.LayerNorm, RMSNorm) for k in kinds) and _are(kinds, dtype, mods)


# the kinds' own forward, and which parameters they have (host.plain)
_PLAIN = {nn.Sequential: (nn.Sequential.forward, 0), nn.GELU: (nn.GELU.forward, 0), nn.Linear: (nn.Linear.forward, 1),
          RMSNorm: (RMSNorm.forward, 2), nn.LayerNorm: (nn.LayerNorm.forward, 3)}     # (and the layers below)


class _Packed(nn.Module):
    """A module whose linear layers of one input (`packed`) keep their weights one below the other in one storage, so
    that a single product serves them.  The layers own their parameters as ever: updates in place are seen, and where
    a parameter has moved to a storage of its own the product falls apart into one per layer.  The rows are padded to
    a multiple of 64, so that every row of the output keeps the alignment that fast products want."""

    packed: tuple = ()
    _whole = None                                     # (weight, bias) over the parameters' common storage

    def _apply(self, fn, *args, **kwargs):
        super()._apply(fn, *args, **kwargs)
        mods = [getattr(self, n) for n in self.packed]
        if all(type(m) is nn.Linear for m in mods):
            params = [m._parameters.get(n) for n in ("weight", "bias") for m in mods]
            if all(type(p) is nn.Parameter and p.is_cuda for p in params) and len(set(map(id, params))) == len(params) \
                    and len({(p.dtype, p.device) for p in params}) == 1 and len({m.in_features for m in mods}) == 1 \
                    and self._joined(mods) is None:
                self._pack(params[:len(mods)], params[len(mods):])
        return self

    def _pack(self, *kinds):
        """Moves the weights, and the biases, one below the other."""
        whole = []
        for parts in kinds:
            pad = -sum(p.shape[0] for p in parts) % 64
            t = torch.cat([p.data for p in parts] + [parts[0].data.new_zeros(pad, *parts[0].shape[1:])])
            at = 0
            for p in parts:
                p.data = t[at:at + p.shape[0]]
                at += p.shape[0]
            whole.append(t)
        self._whole = tuple(whole)

    def _joined(self, mods):
        """_whole, if the parameters still lie in it."""
        if self._whole is not None and not host.joined(tuple(mods), self._whole, nn.Parameter):
            self._whole = None
        return self._whole

    def project(self, x: torch.Tensor):
        """The layers' outputs of x [.., d] (views of one tensor where the weights lie together)."""
        mods = [self._modules[n] for n in self.packed]
        joined = self._joined(mods)
        if joined is None:
            return [F.linear(x, m.weight, m.bias) for m in mods]
        widths = [m.out_features for m in mods]
        return F.linear(x, *joined).split_with_sizes(widths + [joined[0].shape[0] - sum(widths)], -1)[:len(mods)]


_ATTN = (nn.Linear,) * 4 + (RMSNorm,) * 2
_CROSS = (nn.Linear,) * 2 + (RMSNorm,) * 2


class NSASelfAttention(_Packed):
    """The rollout branch of CausalNSSelfAttention over a BlockKVCache."""

    packed = ("q", "k", "v", "g_proj")

    def __init__(self, shape: WanShape, plan: RolloutPlan, layer_idx: int):
        super().__init__()
        d, h = shape.dim, shape.num_heads
        self.h, self.hd, self.plan, self.layer_idx = h, d // h, plan, layer_idx
        self.q, self.k, self.v, self.o = (nn.Linear(d, d) for _ in range(4))
        self.norm_q, self.norm_k = RMSNorm(d, shape.eps), RMSNorm(d, shape.eps)
        self.g_proj = nn.Linear(d, 3 * h)
        nn.init.normal_(self.g_proj.weight, mean=0.0, std=1e-3)     # gates start at 0.5 (initialize_gate, :164-168)
        nn.init.zeros_(self.g_proj.bias)

    def forward(self, x, cache: BlockKVCache, rope: RopeSpec, start_token: int, timer=_NO_TIMER):
        p = self.plan
        B, S, _ = x.shape
        if B != 1:                                    # before anything is projected or appended
            raise NSABackendError(f"the block caches serve batch size 1, got activations {tuple(x.shape)}")
        H, D = self.h, self.hd
        scale = D ** -0.5
        norms = self._modules["norm_q"], self._modules["norm_k"]
        # (one eps serves both norms)
        if _fused(x) and D % 8 == 0 and 32 % (D // 8) == 0 and \
                _are(_ATTN, x.dtype, (*(self._modules[n] for n in self.packed), *norms)) and norms[0].eps == norms[1].eps:
            with timer("qkv_gate_proj"):
                q, k, v, g = self.project(x[0])
                g = g.view(1, S, H, 3)
            # norm and rotary embedding of queries and keys in one pass; the keys stay where they are
            with timer("rope_q"):
                qr = host.qk_norm_rope(q, k, self.norm_q.weight, self.norm_k.weight, self.norm_q.eps, H,
                                       rope.native(x.device, D)).unsqueeze(0)
            with timer("cache_append"):
                cache.append(k.view(S, H, D), v.view(S, H, D), pos0=start_token)
        else:
            with timer("qkv_gate_proj"):
                q = self.norm_q(self.q(x)).view(S, H, D)
                k = self.norm_k(self.k(x)).view(S, H, D)
                v = self.v(x).view(S, H, D)
                g = self.g_proj(x).view(1, S, H, 3)
            # query rotary embedding; the keys receive theirs on the way into the pages, where they are also
            # pooled: one kernel replaces rope + four cache updates + two poolings of the reference layer
            with timer("rope_q"):
                qr = rope_apply(q, rope).unsqueeze(0)
            with timer("cache_append"):
                cache.append(k, v, pos0=start_token, rope=rope)
        nb = cache.n_blocks
        # compressed branch: attention over the pooled history, a dense [1, nb, H, D] view of the pooled
        # keys / values taken as one range of blocks
        with timer("cmp"):
            o_cmp, _ = ops.range_fwd(qr, ops.DenseKV(cache.pooled_keys(), cache.pooled_values()), 0,
                                     -(-nb // p.block), p.block, scale)
        # sliding-window branch: the pages of the last window_chunks chunks through the block table
        with timer("swa"):
            first_tok = max(0, start_token - (p.window_chunks - 1) * S)
            first_blk = first_tok // p.block
            o_swa, _ = ops.range_fwd(qr, cache.kv_source(), first_blk, nb - first_blk, p.block, scale)
        # selection branch
        q_chunk = start_token // S
        if p.progressive_exclude or should_use_selection_attention(nb * p.block, S, p.exclude_window_chunks, 0, causal=False):
            with timer("slc_topk"):
                qp = ops.pool_rows(qr, p.group)
                idx = ops.topk(qp, cache.pooled_keys(), p.topk, scale, p.block, S, S, False,
                               ex_win=p.exclude_window_chunks, prog_excl=p.progressive_exclude,
                               q_chunk_offset=q_chunk, q_group_size=p.group)
            with timer("slc_touch_fetch"):
                cache.touch(idx)
            with timer("slc_attn"):
                o_slc, _ = ops.sel_fwd(qr, cache.kv_source(), idx, p.block, 1, scale, False, p.group)
        else:
            o_slc = torch.zeros_like(qr)
        with timer("gate_sum_oproj"):
            y = ops.gate_combine(g, o_cmp, o_slc, o_swa)
            out = self.o(y.view(1, S, H * D))
        return out


class CrossAttention(_Packed):
    packed = ("k", "v")

    def __init__(self, shape: WanShape):
        super().__init__()
        d, h = shape.dim, shape.num_heads
        self.h, self.hd = h, d // h
        self.q, self.k, self.v, self.o = (nn.Linear(d, d) for _ in range(4))
        self.norm_q, self.norm_k = RMSNorm(d, shape.eps), RMSNorm(d, shape.eps)

    def forward(self, x, context):
        B, S, d = x.shape
        L = context.shape[1]
        if _fused(x) and context.dtype == x.dtype and \
                _are(_CROSS, x.dtype, tuple(self._modules[n] for n in ("k", "v", "norm_q", "norm_k"))):
            heads = lambda t: t.unflatten(-1, (self.h, self.hd)).transpose(1, 2)
            k, v = self.project(context)
            q = heads(host.rms_rows(self.q(x), self.norm_q.weight, self.norm_q.eps))
            k = heads(host.rms_rows(k, self.norm_k.weight, self.norm_k.eps))
            y = F.scaled_dot_product_attention(q, k, heads(v))
            return self.o(y.transpose(1, 2).reshape(B, S, d))
        q = self.norm_q(self.q(x)).view(B, S, self.h, self.hd).transpose(1, 2)
        k = self.norm_k(self.k(context)).view(B, L, self.h, self.hd).transpose(1, 2)
        v = self.v(context).view(B, L, self.h, self.hd).transpose(1, 2)
        y = F.scaled_dot_product_attention(q, k, v)
        return self.o(y.transpose(1, 2).reshape(B, S, self.h * self.hd))


_NO_VECTOR = (None, None)


class Block(nn.Module):
    def __init__(self, shape: WanShape, plan: RolloutPlan, layer_idx: int):
        super().__init__()
        d = shape.dim
        self.eps = shape.eps
        self.self_attn = NSASelfAttention(shape, plan, layer_idx)
        self.norm3 = nn.LayerNorm(d, eps=shape.eps)
        self.cross_attn = CrossAttention(shape)
        self.ffn = nn.Sequential(nn.Linear(d, shape.ffn_dim), nn.GELU(approximate="tanh"), nn.Linear(shape.ffn_dim, d))
        self.modulation = nn.Parameter(torch.randn(1, 6, d) / d ** 0.5)

    def fusable(self, dtype: torch.dtype) -> bool:
        own = self._modules
        attn, cross, ffn = own["self_attn"], own["cross_attn"], own["ffn"]
        if len(ffn._modules) != 3:
            return False
        up, act, down = ffn._modules.values()
        return _are(_BLOCK, dtype, (self, attn, cross, ffn, act, up, down, own["norm3"], attn._modules.get("o"), cross._modules.get("o"))) \
            and act.approximate == "tanh" and up._parameters.get("bias") is not None and _row(self.modulation, dtype)

    def fused(self, x, pending, e, context, cache, rope, start_token, timer=_NO_TIMER):
        """forward() with the residual of the sub-layer in front still `pending` (its output and gate vector, or
        None): returns (x, pending) for the next block.  e: the six fp32 rows of the time modulation."""
        m = self.modulation[0].unbind(0)
        vec = lambda i: (m[i], e[i])
        y, gate = pending if pending is not None else (None, _NO_VECTOR)
        with timer("norm_modulation"):
            x, h = host.residual_norm(x, y, gate, vec(1), vec(0), True, True, self.eps)
        y = self.self_attn(h, cache, rope, start_token, timer)
        with timer("norm_modulation"):
            x, h = host.residual_norm(x, y, vec(2), (self.norm3.weight, None), (self.norm3.bias, None), False, True,
                                      self.norm3.eps)
        with timer("cross_attn"):
            y = self.cross_attn(h, context)
        with timer("norm_modulation"):
            x, h = host.residual_norm(x, y, _NO_VECTOR, vec(4), vec(3), True, True, self.eps)
        with timer("ffn"):
            up, down = self.ffn[0], self.ffn[2]
            h = torch._addmm_activation(up.bias, h[0], up.weight.t(), use_gelu=True)     # tanh form, in the epilogue
            y = F.linear(h, down.weight, down.bias).unsqueeze(0)
        return x, (y, vec(5))

    def forward(self, x, e0, context, cache, rope, start_token, timer=_NO_TIMER):
        e = (self.modulation.float() + e0).unbind(1)                 # six [1, dim] rows (fp32, as the reference)
        d = x.shape[-1]
        with timer("norm_modulation"):
            h = (F.layer_norm(x.float(), (d,), eps=self.eps) * (1 + e[1]) + e[0]).to(x.dtype)
        y = self.self_attn(h, cache, rope, start_token, timer)
        with timer("norm_modulation"):
            x = x + (y.float() * e[2]).to(x.dtype)
        with timer("cross_attn"):
            x = x + self.cross_attn(self.norm3(x), context)
        with timer("ffn"):
            h = (F.layer_norm(x.float(), (d,), eps=self.eps) * (1 + e[4]) + e[3]).to(x.dtype)
            x = x + (self.ffn(h).float() * e[5]).to(x.dtype)
        return x


_PLAIN.update((c, (c.forward, 0)) for c in (NSASelfAttention, CrossAttention, Block))
_BLOCK = (Block, NSASelfAttention, CrossAttention, nn.Sequential, nn.GELU, nn.Linear, nn.Linear, nn.LayerNorm, nn.Linear, nn.Linear)


class CausalWanNSA(nn.Module):
    def __init__(self, shape: WanShape, plan: RolloutPlan):
        super().__init__()
        self.shape, self.plan = shape, plan
        d = shape.dim
        self.patch_embedding = nn.Conv3d(shape.in_dim, d, kernel_size=shape.patch, stride=shape.patch)
        self.text_embedding = nn.Sequential(nn.Linear(shape.text_dim, d), nn.GELU(approximate="tanh"), nn.Linear(d, d))
        self.time_embedding = nn.Sequential(nn.Linear(shape.freq_dim, d), nn.SiLU(), nn.Linear(d, d))
        self.time_projection = nn.Sequential(nn.SiLU(), nn.Linear(d, 6 * d))
        self.blocks = nn.ModuleList([Block(shape, plan, i) for i in range(shape.num_layers)])
        self.head_norm_eps = shape.eps
        self.head = nn.Linear(d, shape.out_dim * math.prod(shape.patch))
        self.head_modulation = nn.Parameter(torch.randn(1, 2, d) / d ** 0.5)
        hd = d // shape.num_heads
        self.register_buffer("_dummy", torch.zeros(1), persistent=False)
        self.freqs = torch.cat([rope_table(1024, hd - 4 * (hd // 6)), rope_table(1024, 2 * (hd // 6)),
                                rope_table(1024, 2 * (hd // 6))], dim=1)
        self._rope = None                        # the last RopeSpec: its device tables serve the next forward

    def forward(self, latents, t, context_embedded, start_frame, caches: List[BlockKVCache], timer=_NO_TIMER):
        """latents [1, C, f, h, w]; t scalar timestep; returns the prediction in latent layout."""
        sh = self.shape
        x = self.patch_embedding(latents)
        _, _, f, gh, gw = x.shape
        x = x.flatten(2).transpose(1, 2).contiguous()
        S = x.shape[1]
        temb = sinusoidal_embedding(sh.freq_dim, torch.full((1,), float(t), device=x.device)).to(x.dtype)
        e = self.time_embedding(temb)
        e0 = self.time_projection(e).float().view(1, 6, sh.dim)
        rope = self._rope = RopeSpec(self.freqs, (gh, gw), start_frame, (1, 1, 1), like=self._rope)
        start_token = start_frame * gh * gw
        if _fused(x) and _row(self.head_modulation, x.dtype) and all(type(b) is Block and b.fusable(x.dtype) for b in self.blocks):
            pending, e_rows = None, e0[0].unbind(0)
            for blk, cache in zip(self.blocks, caches):
                x, pending = blk.fused(x, pending, e_rows, context_embedded, cache, rope, start_token, timer)
            m, ef = self.head_modulation[0].unbind(0), e[0].float()
            y, gate = pending if pending is not None else (None, _NO_VECTOR)
            _, x = host.residual_norm(x, y, gate, (m[1], ef), (m[0], ef), True, True, self.head_norm_eps)
            return self._unpatch(self.head(x), f, gh, gw)
        for blk, cache in zip(self.blocks, caches):
            x = blk(x, e0, context_embedded, cache, rope, start_token, timer)
        m = (self.head_modulation.float() + e.float().unsqueeze(1)).unbind(1)
        x = (F.layer_norm(x.float(), (sh.dim,), eps=self.head_norm_eps) * (1 + m[1]) + m[0]).to(x.dtype)
        return self._unpatch(self.head(x), f, gh, gw)

    def _unpatch(self, x, f, gh, gw):
        """[1, S, out * pf*ph*pw] -> latent layout"""
        sh = self.shape
        pf, ph, pw = sh.patch
        x = x.view(1, f, gh, gw, pf, ph, pw, sh.out_dim).permute(0, 7, 1, 4, 2, 5, 3, 6)
        return x.reshape(1, sh.out_dim, f * pf, gh * ph, gw * pw)


def make_caches(shape: WanShape, plan: RolloutPlan, device) -> List[BlockKVCache]:
    """One page pool per layer.  Without a cap every block of the rollout is resident.  With one the
    pool holds cache_cap_frames frames' worth of blocks per head (at least the protected window and
    the chunk being written) PLUS room for the blocks one call can select (top-k x query groups per
    head): a call needs its window and everything it selected resident at the same time, and with
    random weights the selections of the 74 query groups hardly overlap.  The rest of the history
    lives in the pinned host tier and comes back when selected."""
    gh, gw = plan.latent_h // shape.patch[1], plan.latent_w // shape.patch[2]
    tokens = plan.latent_frames * gh * gw
    max_blocks = -(-tokens // plan.block)
    H, D = shape.num_heads, shape.dim // shape.num_heads
    chunk_blocks = -(-plan.frames_per_chunk * gh * gw // plan.block) + 1
    protect = plan.window_chunks * chunk_blocks                     # the window and the chunk being written stay resident
    if plan.cache_cap_frames is None:
        pages, host = H * max_blocks, False
    else:
        groups = -(-plan.frames_per_chunk * gh * gw // plan.group)
        pages = H * (max(-(-plan.cache_cap_frames * gh * gw // plan.block), protect + chunk_blocks) + plan.topk * groups)
        host = True
    return [BlockKVCache(H, D, pages, max_blocks, plan.block, torch.bfloat16, device, host_tier=host, protect_blocks=protect)
            for _ in range(shape.num_layers)]


@dataclass
class RolloutResult:
    seconds: float
    latent_frames: int
    forwards: int
    frames_per_second: float
    cache: dict = field(default_factory=dict)
    latents: Optional[torch.Tensor] = None


@torch.no_grad()
def rollout(model: CausalWanNSA, caches: List[BlockKVCache], plan: RolloutPlan, device, keep_latents: bool = False,
            timer=_NO_TIMER) -> RolloutResult:
    """The denoising loop of CausalWanT2VPipeline.generate (pipeline_wan_causal.py:349-495): per chunk,
    len(timesteps) denoising forwards (each rewrites the chunk's K/V in the caches), then one forward
    of the clean chunk at t = 0 that leaves the final K/V behind.  Returns the wall time of the loop
    (the reference's "Denoising Time") and latent frames per second."""
    sh = model.shape
    gen = torch.Generator(device=device).manual_seed(plan.seed)
    noise = torch.randn(1, sh.in_dim, plan.latent_frames, plan.latent_h, plan.latent_w, generator=gen, device=device,
                        dtype=torch.bfloat16)

    def new_context():
        raw = torch.randn(1, sh.text_len, sh.text_dim, generator=gen, device=device, dtype=torch.bfloat16)
        return model.text_embedding(raw)

    context = new_context()
    next_switch = plan.new_prompt_every
    latents = torch.zeros_like(noise) if keep_latents else None
    for c in caches:
        c.reset()
    forwards = 0
    torch.cuda.synchronize(device)
    t0 = time.perf_counter()
    for start in range(0, plan.latent_frames, plan.frames_per_chunk):
        if next_switch is not None and start >= next_switch:
            context = new_context()
            next_switch += plan.new_prompt_every
        x_t = noise[:, :, start:start + plan.frames_per_chunk]
        x0 = x_t
        for i, t in enumerate(plan.timesteps):
            sigma = t / 1000.0
            v = model(x_t, t, context, start, caches, timer)
            forwards += 1
            x0 = (x_t.float() - sigma * v.float()).to(x_t.dtype)               # flow prediction -> clean estimate
            if i + 1 < len(plan.timesteps):
                s2 = plan.timesteps[i + 1] / 1000.0
                eps = torch.randn(x0.shape, generator=gen, device=device, dtype=x0.dtype)
                x_t = ((1.0 - s2) * x0.float() + s2 * eps.float()).to(x0.dtype)
        if latents is not None:
            latents[:, :, start:start + plan.frames_per_chunk] = x0
        model(x0, 0.0, context, start, caches, timer)                          # cache-write forward on the clean chunk
        forwards += 1
    torch.cuda.synchronize(device)
    dt = time.perf_counter() - t0
    stats = {"hits": 0, "misses": 0, "pages_evicted": 0, "pages_fetched": 0, "bytes_to_host": 0, "bytes_from_host": 0}
    for c in caches:
        c.check_status()
        s = c.stats()
        for k in stats:
            stats[k] += s[k]
    total = stats["hits"] + stats["misses"]
    stats["hit_rate"] = stats["hits"] / total if total else 0.0
    return RolloutResult(dt, plan.latent_frames, forwards, plan.latent_frames / dt, stats, latents)


def build(shape: WanShape, plan: RolloutPlan, device, seed: int = 0):
    torch.manual_seed(seed)
    model = CausalWanNSA(shape, plan).to(device=device, dtype=torch.bfloat16).eval()
    return model, make_caches(shape, plan, device)
