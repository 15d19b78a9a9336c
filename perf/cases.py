"""The work that users of this package have it do, as cases that can be timed.

Six kinds of pass, each through the public entry points and over the sizes they are used at:

  attend    inference over dense K/V: pool the keys, select blocks, selection attention
  train     one training pass of the sparse branch: selection, selection attention, gated sum of the
            three branches, and the gradients of everything that is differentiable
  step      the operators of one forward + backward step captured once in a CUDA graph and replayed
  memory    selection and attention over a memory far longer than the queries (single rank)
  generate  one denoising forward of the chunk-by-chunk video transformer over its block caches
  recall    one layer's cache work in long rolling generation, with evicted blocks fetched back
"""
import math

import torch

from omnimem_b200 import ops, rollout
from omnimem_b200.cache import BlockKVCache, RopeSpec, rope_apply
from omnimem_b200.graph import CapturedStep
from omnimem_b200.nsa.ops import gated_branch_sum, parallel_nsa_topk_grouped_heads, selection_attention
from omnimem_b200.sharded import ShardedSelection

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # One latent frame of a 240x416 video against the four frames before it: the smallest call that a
        # generation makes, where the host's work and the launches count.
        dict(name="attend small", kind="attend", dtype="bf16", B=1, M=390, N=1560, H=12, D=128, block=64, group=64,
             topk=8, chunk=390, offset=3, kv_heads=12),
        # One 480x832 frame against four, fp32 tensors: the operator-level configuration in fp32.
        dict(name="attend frame fp32", kind="attend", dtype="fp32", B=1, M=1560, N=6240, H=12, D=128, block=64,
             group=64, topk=16, chunk=1560, offset=3, kv_heads=12),
        # A three-frame chunk against the whole 21-frame clip with blocks of one 15 x 2 spatial tile and
        # groups of half a tile.
        dict(name="attend tiles 30/15", kind="attend", dtype="bf16", B=1, M=4680, N=32760, H=12, D=128, block=30,
             group=15, topk=16, chunk=4680, offset=6, kv_heads=12),
        # Training on one chunk against the clip, 64-token blocks: eager autograd.
        dict(name="train chunk 64/64", kind="train", dtype="bf16", B=1, M=4680, N=32760, H=12, D=128, block=64,
             group=64, topk=16, chunk=4680, offset=6, kv_heads=12),
        # Training on a whole 21-frame clip, chunk-causal, 15 x 2 tiles: the largest pass.
        dict(name="train clip 30/15", kind="train", dtype="bf16", B=1, M=32760, N=32760, H=12, D=128, block=30,
             group=15, topk=16, chunk=4680, offset=0, kv_heads=12),
        # 24-token blocks (6 x 4 tiles), top-64, fp16, 64-wide heads that share selections in groups of four.
        dict(name="train 24/12 fp16 d64", kind="train", dtype="fp16", B=2, M=3120, N=3120, H=16, D=64, block=24,
             group=12, topk=64, chunk=1560, offset=0, kv_heads=4),
        # The operators of one step on the clip, replayed as a graph: device time without the host.
        dict(name="step 64/64", kind="step", dtype="bf16", B=1, M=4680, N=32760, H=12, D=128, block=64, group=64,
             topk=16, chunk=1560, offset=18),
        # A million-token memory read by one chunk.
        dict(name="memory 1M", kind="memory", dtype="bf16", B=1, M=4680, N=1048576, H=12, D=128, block=64, group=64,
             topk=16, chunk=4680, offset=221),
        # The transformer's forward (six of its blocks): the first single-frame chunk of a 240x416 video, the
        # first chunk of a 480x832 one, and the last chunk of a 21-frame one.
        dict(name="generate small", kind="generate", layers=6, h=30, w=52, frames=1, start=0),
        dict(name="generate first chunk", kind="generate", layers=6, h=60, w=104, frames=3, start=0),
        dict(name="generate last chunk", kind="generate", layers=6, h=60, w=104, frames=3, start=18),
        # Rolling generation at 240x416: 240 frames of history, 24 frames' worth of pages (and the blocks one
        # call can select) resident.
        dict(name="recall rolling", kind="recall", H=12, h=30, w=52, frames=3, history=240, resident=24, topk=16),
    ]


# ------------------------------------------------------------------------------------------ other cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    w = work(case)
    return w["bytes"] / 6e12 + w["flops"] / 6e14


def _draw(rng):
    kind = rng.choice(("attend", "attend", "train", "train", "step", "memory", "generate", "generate", "recall"))
    if kind == "generate":
        frames = rng.randint(1, 3)
        return dict(kind=kind, layers=rng.randint(2, 6), h=2 * rng.randint(8, 30), w=2 * rng.randint(12, 52),
                    frames=frames, start=frames * rng.randint(0, 18 // frames))
    if kind == "recall":
        frames = rng.randint(1, 3)
        return dict(kind=kind, H=rng.choice((8, 12, 16)), h=2 * rng.randint(8, 15), w=2 * rng.randint(14, 26),
                    frames=frames, history=frames * rng.randint(60 // frames, 240 // frames),
                    resident=rng.randint(9, 24), topk=rng.choice((8, 16)))
    if kind == "memory":
        M = rng.randint(400, 4680)
        N = _log_int(rng, 65536, 1048576)
        return dict(kind=kind, dtype="bf16", B=1, M=M, N=N, H=12, D=128, block=64, group=64, topk=rng.choice((8, 16, 24)),
                    chunk=M, offset=N // M)
    if kind == "step":
        M = _log_int(rng, 400, 4680)
        N = _log_int(rng, M, 32760)
        return dict(kind=kind, dtype="bf16", B=1, M=M, N=N, H=12, D=128, block=64, group=64, topk=rng.choice((8, 16)),
                    chunk=M, offset=N // M)
    block, group = rng.choice(((64, 64), (64, 64), (30, 15), (30, 15), (60, 60), (24, 12)))
    D = rng.choice((128, 128, 64))
    H = rng.choice((12, 12, 16, 8))
    frame = block * rng.randint(4, 52)                        # tokens of one chunk, whole blocks of them
    chunks = rng.randint(2, 21)
    whole = kind == "train" and rng.random() < 0.5            # all chunks at once, or the last one against all
    return dict(kind=kind, dtype=rng.choice(("bf16", "bf16", "bf16", "fp16", "fp32")), B=rng.choice((1, 1, 2)),
                M=frame * chunks if whole else frame, N=frame * chunks, H=H, D=D, block=block, group=group,
                topk=rng.choice((8, 16, 16, 64 if block < 64 else 24)), chunk=frame, offset=0 if whole else chunks - 1,
                kv_heads=rng.choice((H, H, H // 4)))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= most:
            return case


# --------------------------------------------------------------------------------------------- the state
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, _generator(seed), seed)


def run(state):
    return state["run"](state)


def _qkv(case, gen):
    dt = DTYPES[case["dtype"]]
    B, M, N, H, D = (case[x] for x in ("B", "M", "N", "H", "D"))
    rand = lambda n: torch.randn(B, n, H, D, generator=gen, device="cuda", dtype=dt)
    return rand(M), rand(N), rand(N)


def _select(case, q, k):
    kp = ops.pool_rows(k, case["block"])
    return parallel_nsa_topk_grouped_heads(q, kp, case["kv_heads"], case["topk"], case["block"], case["chunk"],
                                           causal=True, group_size=case["group"], q_chunk_offset=case["offset"],
                                           allow_ragged=True)


def _prepare_attend(case, gen, seed):
    q, k, v = _qkv(case, gen)
    return dict(run=_run_attend, case=case, q=q, k=k, v=v)


def _run_attend(s):
    c = s["case"]
    with torch.no_grad():
        idx = _select(c, s["q"], s["k"])
        out, lse = selection_attention(s["q"], s["k"], s["v"], idx, c["topk"], c["block"], chunk_size=c["chunk"],
                                       causal=False, return_lse=True, group_size=c["group"], allow_ragged=True)
    return out, lse, idx


def _prepare_train(case, gen, seed):
    q, k, v = (t.requires_grad_(True) for t in _qkv(case, gen))
    like_q = lambda: torch.randn(q.shape, generator=gen, device="cuda", dtype=q.dtype)
    s = dict(run=_run_train, case=case, q=q, k=k, v=v, upstream=like_q())
    if case["dtype"] != "fp32":                               # the gated sum is a 16-bit operator
        s["compressed"], s["window"] = like_q().requires_grad_(True), like_q().requires_grad_(True)
        s["gates"] = torch.randn(*q.shape[:3], 3, generator=gen, device="cuda", dtype=q.dtype).requires_grad_(True)
    return s


def _run_train(s):
    c = s["case"]
    with torch.no_grad():
        idx = _select(c, s["q"], s["k"])
    x = selection_attention(s["q"], s["k"], s["v"], idx, c["topk"], c["block"], chunk_size=c["chunk"],
                            causal=c["offset"] == 0, group_size=c["group"], allow_ragged=True)
    leaves = [s["q"], s["k"], s["v"]]
    if "gates" in s:
        x = gated_branch_sum(s["gates"], s["compressed"], x, s["window"])
        leaves += [s["gates"], s["compressed"], s["window"]]
    return (x.detach(), idx) + torch.autograd.grad(x, leaves, s["upstream"])


def _prepare_step(case, gen, seed):
    q, k, v = _qkv(case, gen)
    upstream = torch.randn(q.shape, generator=gen, device="cuda", dtype=q.dtype)
    scale, kv = case["D"] ** -0.5, ops.DenseKV(k, v)

    def step():
        idx, _, _ = ops.select_blocks(q, k, case["topk"], scale, case["block"], case["group"], case["chunk"],
                                      case["chunk"], True, q_chunk_offset=case["offset"])
        out, lse = ops.sel_fwd(q, kv, idx, case["block"], 1, scale, False, case["group"])
        dq, dk, dv = ops.sel_bwd(q, kv, idx, out, lse, upstream, case["block"], 1, scale, False, case["group"])
        return idx, out, lse, dq, dk, dv

    return dict(run=_run_step, inputs=(q, k, v, upstream), step=CapturedStep(step))


def _run_step(s):
    return s["step"].replay()


def _prepare_memory(case, gen, seed):
    q, k, v = _qkv(case, gen)
    return dict(run=_run_memory, case=case, q=q, k=k, v=v, selection=ShardedSelection())


def _run_memory(s):
    c = s["case"]
    return s["selection"].forward(s["q"], s["k"], s["v"], c["topk"], c["block"], c["group"], c["chunk"], True,
                                  q_chunk_offset=c["offset"])


def _prepare_generate(case, gen, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    shape = rollout.WanShape(num_layers=case["layers"])
    plan = rollout.RolloutPlan(latent_frames=case["start"] + case["frames"], frames_per_chunk=case["frames"],
                               latent_h=case["h"], latent_w=case["w"])
    with torch.device(dev):                                   # the random weights are drawn on the device: faster
        model, caches = rollout.build(shape, plan, dev, seed)
    model.freqs = model.freqs.cpu()                           # where build() leaves the rotary table
    rand = lambda *s: torch.randn(*s, generator=gen, device=dev, dtype=torch.bfloat16)
    history = case["start"] * (case["h"] // 2) * (case["w"] // 2)
    if history:
        for cache in caches:
            cache.append(rand(history, shape.num_heads, 128), rand(history, shape.num_heads, 128))
    with torch.no_grad():
        context = model.text_embedding(rand(1, shape.text_len, shape.text_dim))
    latents = rand(1, shape.in_dim, case["frames"], case["h"], case["w"])
    return dict(run=_run_generate, case=case, model=model, caches=caches, context=context, latents=latents)


def _run_generate(s):
    with torch.no_grad():
        y = s["model"](s["latents"], 750.0, s["context"], s["case"]["start"], s["caches"])
    return [y] + [t for c in s["caches"] for t in (c.k_pooled, c.v_pooled)]


def _recall_sizes(case):
    chunk = case["frames"] * (case["h"] // 2) * (case["w"] // 2)
    per_frame = chunk // case["frames"]
    groups = -(-chunk // 64)
    max_blocks = -(-(case["history"] + case["frames"]) * per_frame // 64)
    window = 3 * (groups + 1)
    pages = case["H"] * (max(-(-case["resident"] * per_frame // 64), window + groups + 1) + case["topk"] * groups)
    return chunk, groups, max_blocks, window, pages


def _prepare_recall(case, gen, seed):
    chunk, groups, max_blocks, window, pages = _recall_sizes(case)
    H, D = case["H"], 128
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda", dtype=torch.bfloat16)
    cache = BlockKVCache(H, D, pages, max_blocks, host_tier=True, protect_blocks=window)
    for _ in range(case["history"] // case["frames"]):
        cache.append(rand(chunk, H, D), rand(chunk, H, D))
    freqs = torch.cat([rollout.rope_table(1024, D - 4 * (D // 6)), rollout.rope_table(1024, 2 * (D // 6)),
                       rollout.rope_table(1024, 2 * (D // 6))], dim=1)
    rope = RopeSpec(freqs, (case["h"] // 2, case["w"] // 2), case["history"])
    # the queries of four denoising steps: each asks for blocks of its own
    return dict(run=_run_recall, case=case, cache=cache, rope=rope, start=cache.n_tokens, at=0,
                q=[rand(chunk, H, D) for _ in range(4)], k=rand(chunk, H, D), v=rand(chunk, H, D))


def _run_recall(s):
    c, cache = s["case"], s["cache"]
    q = rope_apply(s["q"][s["at"] % 4], s["rope"]).unsqueeze(0)
    s["at"] += 1
    chunk = q.shape[1]
    cache.append(s["k"], s["v"], pos0=s["start"], rope=s["rope"])
    idx = ops.topk(ops.pool_rows(q, 64), cache.pooled_keys(), c["topk"], 128 ** -0.5, 64, chunk, chunk, False, ex_win=3,
                   prog_excl=True, q_chunk_offset=s["start"] // chunk, q_group_size=64)
    out, lse = cache.selection_attention(q, idx, return_lse=True)
    return out, lse, idx, cache.k_pooled, cache.v_pooled, cache.counters


_PREPARE = {"attend": _prepare_attend, "train": _prepare_train, "step": _prepare_step, "memory": _prepare_memory,
            "generate": _prepare_generate, "recall": _prepare_recall}


# ------------------------------------------------------------------------------- what cannot be avoided
def _seen_keys(case):
    """Keys that one query attends, summed over the queries of one head."""
    M, N, chunk, block, T = (case[x] for x in ("M", "N", "chunk", "block", "topk"))
    total = 0
    for c in range(-(-M // chunk)):
        rows = min(chunk, M - c * chunk)
        total += rows * min(T * block, N, (c + case["offset"] + 1) * chunk)
    return total


def work(case):
    if case["kind"] == "generate":
        return _work_generate(case)
    if case["kind"] == "recall":
        chunk, groups, max_blocks, _, _ = _recall_sizes(case)
        H, row = case["H"], case["H"] * 128 * 2
        picked = min(groups * case["topk"], max_blocks)
        # q, k, v in; k, v into the pages; out; the pooled keys; each head's selected blocks' k and v
        return {"bytes": 6 * chunk * row + max_blocks * row + 2 * picked * 64 * row,
                "flops": 4 * 128 * H * chunk * min(case["topk"] * 64, max_blocks * 64)}
    B, M, N, H, D = (case[x] for x in ("B", "M", "N", "H", "D"))
    esz = 4 if case["dtype"] == "fp32" else 2
    row = H * D * esz
    groups = -(-M // case["group"])
    ids = groups * H * case["topk"] * 4
    picked = min(N, groups * case["topk"] * case["block"])     # tokens of V that are read for at least one query
    flops = 4 * D * H * B * _seen_keys(case)
    if case["kind"] in ("attend", "memory"):
        return {"bytes": B * (row * (2 * M + N + picked) + 4 * H * M + ids), "flops": flops}
    # forward, and in the backward dQ, dK, dV, dP and the scores again; dK and dV of every token
    bytes_ = B * (row * (5 * M + 2 * N + 2 * N) + 4 * H * M + ids)
    if case["kind"] == "train" and case["dtype"] != "fp32":    # gates and two more branches, and their gradients
        bytes_ += B * (row * 4 * M + 4 * 3 * M * H * esz)
    return {"bytes": bytes_, "flops": 3.5 * flops}


def _work_generate(case):
    s = rollout.WanShape(num_layers=case["layers"])
    S = case["frames"] * (case["h"] // 2) * (case["w"] // 2)
    start = case["start"] * (case["h"] // 2) * (case["w"] // 2)
    d, f, L, H = s.dim, s.ffn_dim, s.num_layers, s.num_heads
    total = start + S
    blocks = -(-total // 64)
    window = total - max(0, start - 2 * S) // 64 * 64
    hidden = 3 * S // 64 if start >= 3 * S else 0              # what the window covers is not selected again
    selected = min(16, max(0, blocks - hidden)) * 64
    linear = S * (6 * d * d + 3 * H * d + 2 * d * f) + s.text_len * 2 * d * d
    attended = S * (blocks + window + min(selected, total) + s.text_len)
    weights = 8 * d * d + 3 * H * d + 2 * d * f
    io = 2 * s.in_dim * case["frames"] * case["h"] * case["w"] * 2
    return {"bytes": 2 * L * weights + io + L * 2 * 2 * d * (S + window + blocks) + 2 * s.text_len * d,
            "flops": 2.0 * L * linear + 4.0 * L * d * attended + 2.0 * S * d * 2 * 64}


def tolerance(case):
    if case["kind"] == "generate":
        # bf16 roundings of up to six blocks in a row, and selections whose scores all but tie (the same
        # forward with the window's blocks listed one by one is 3e-3 away)
        return {"rel": 1e-2, "max": 0.4}
    # bf16 / fp16 operands with fp32 sums; ids may swap where two scores agree to the last bits
    return {"rel": 1e-2, "max": 0.5, "differ": 2e-3}
