"""The work this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values. ``prepare(case, seed)`` makes what a user's program holds before the call,
``run(state)`` is one pass through the public entry points, ``work(case)`` the bytes and operations that pass cannot
do without, ``tolerance(case)`` how far two correct implementations of the same precision may be apart.
``listed()`` are the cases quoted in the documentation, ``draw(rng)`` gives more of the same ranges.

Six kinds of work:

* ``train``     one optimizer step of a Llama-shaped model through ``Trainer.train_step``: tokens from pinned host
                memory, forward, backward over every micro-batch, clipping, sharded AdamW, loss read back;
* ``logits``    evaluation / prefill: ``LlamaModel.logits`` over a batch of sequences;
* ``attention`` ``flash_attention`` as an autograd op inside somebody else's model: forward and backward, or forward
                alone, causal or not, with grouped or one-to-one KV heads;
* ``sparse``    ``SparseRingAttention``: sliding window plus global blocks, forward and backward;
* ``fp8kv``     ``QuantizedRingAttention``: attention over the e4m3 cache format (forward: the format is a serving
                one, it has no gradient of its own on one GPU);
* ``linear``    the bias-free ``linear`` with a residual, forward and backward (the rows are the inner dimension of the weight
                gradient, which the GEMM takes in multiples of 8).
"""
import math

import torch

from zenyx_b200.models import LlamaConfig, LlamaModel
from zenyx_b200.ops.attention import flash_attention
from zenyx_b200.ops.gemm import linear
from zenyx_b200.train import Trainer, TrainerConfig
from zenyx_b200.train.fp8_kv_quantization import QuantizedRingAttention
from zenyx_b200.train.sparse_ring_attention import SparsePattern, SparseRingAttention

HEAD_DIM = 128   # what the attention kernels take


def listed():
    return [
        # the fine-tuning example of this repository: a step is all launches and host work
        dict(name="train_tiny", kind="train", layers=2, d_model=256, heads=2, kv_heads=1, ffn=512, vocab=512,
             batch=2, seq=256),
        # a model of about 0.4 G parameters on 4K contexts: every kernel at a size between tiny and 8B
        dict(name="train_mid", kind="train", layers=4, d_model=2048, heads=16, kv_heads=4, ffn=5632, vocab=32000,
             batch=4, seq=4096),
        # the benchmark's own layer shapes and sequence, with two layers so that a step is a fraction of a second
        dict(name="train_8b_2_layers_32k", kind="train", layers=2, d_model=4096, heads=32, kv_heads=8, ffn=14336,
             vocab=128256, batch=1, seq=32768),
        # evaluation of the 8B layer shapes on two documents of 15 blocks each
        dict(name="logits_8b_2_layers", kind="logits", layers=2, d_model=4096, heads=32, kv_heads=8, ffn=14336,
             vocab=128256, batch=2, seq=1920),
        # attention of one 8K sequence of the 8B shape, as a training step sees it
        dict(name="attention_8k", kind="attention", batch=1, seq=8192, heads=32, kv_heads=8, causal=True, backward=True),
        # the benchmark's sequence length
        dict(name="attention_32k", kind="attention", batch=1, seq=32768, heads=32, kv_heads=8, causal=True,
             backward=True),
        # a small encoder: bidirectional, one KV head per head, an odd number of blocks, bound by launches
        dict(name="attention_small", kind="attention", batch=2, seq=384, heads=8, kv_heads=8, causal=False,
             backward=True),
        # the documented sparse pattern (4096-token window, every 64th block global) over 64K tokens
        dict(name="sparse_64k", kind="sparse", seq=65536, heads=32, kv_heads=8, window=4096, global_every=64),
        # prefill over the e4m3 cache format
        dict(name="fp8kv_16k", kind="fp8kv", batch=1, seq=16384, heads=32, kv_heads=8),
        # a projection of somebody's own model: rows and columns that no tile divides
        dict(name="linear_ragged", kind="linear", rows=3000, inner=2056, outer=5640),
        # the down projection of the 8B shape over two 8K sequences
        dict(name="linear_large", kind="linear", rows=16384, inner=14336, outer=4096),
        # a handful of rows, as a classifier head or an adapter sees them: one wave, latency only
        dict(name="linear_small", kind="linear", rows=64, inner=1024, outer=1024),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(x / step)) * step))


def draw(rng):
    kind = rng.choice(("train", "train", "logits", "attention", "attention", "sparse", "fp8kv", "linear", "linear"))
    if kind in ("train", "logits"):
        heads = rng.choice((2, 4, 8, 12, 16, 24, 32))
        kv = rng.choice([h for h in (1, 2, 4, 8) if heads % h == 0])
        d_model = heads * HEAD_DIM
        c = dict(kind=kind, layers=rng.randint(1, 3), d_model=d_model, heads=heads, kv_heads=kv,
                 ffn=8 * rng.randint(d_model // 6, d_model * 7 // 16), vocab=_log(rng, 512, 65536, 8),
                 batch=rng.randint(1, 4), seq=_log(rng, 256, 8192, 128))
        return c
    if kind == "attention":
        heads = rng.choice((1, 2, 4, 6, 8, 16, 32))
        kv = rng.choice([h for h in (1, 2, 4, 8, 16, 32) if heads % h == 0])
        seq = _log(rng, 128, 16384, 128)
        return dict(kind=kind, batch=rng.randint(1, 4) if seq <= 4096 else 1, seq=seq, heads=heads, kv_heads=kv,
                    causal=rng.random() < 0.75, backward=rng.random() < 0.75)
    if kind == "sparse":
        return dict(kind=kind, seq=_log(rng, 4096, 65536, 128), heads=rng.choice((8, 16, 32)), kv_heads=rng.choice((2, 4, 8)),
                    window=128 * _log(rng, 2, 32), global_every=rng.choice((0, 16, 64)))
    if kind == "fp8kv":
        return dict(kind=kind, batch=rng.randint(1, 3), seq=_log(rng, 256, 16384, 128), heads=rng.choice((8, 16, 32)),
                    kv_heads=rng.choice((2, 4, 8)))
    return dict(kind=kind, rows=_log(rng, 8, 16384, 8), inner=_log(rng, 64, 8192, 8), outer=_log(rng, 64, 8192, 8))


# ------------------------------------------------------------------------------------------------


def _config(c):
    return LlamaConfig(vocab_size=c["vocab"], d_model=c["d_model"], n_layers=c["layers"], n_heads=c["heads"],
                       n_kv_heads=c["kv_heads"], head_dim=HEAD_DIM, ffn_dim=c["ffn"])


def _normal(gen, *shape, std=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).bfloat16()


def _qkv(c, gen, grad):
    # unit-variance heads: what a normalised, projected and rotated activation looks like
    shape = (c.get("batch", 1), c["seq"])
    t = [_normal(gen, *shape, c[h], HEAD_DIM) for h in ("heads", "kv_heads", "kv_heads")]
    return [x.requires_grad_(True) for x in t] if grad else t


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "train":
        host = torch.Generator().manual_seed(seed)
        trainer = Trainer(_config(case), TrainerConfig(lr=3e-4, seq_len=case["seq"], global_batch=case["batch"],
                                                       max_grad_norm=1.0, weight_decay=0.1, seed=seed))
        tokens = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=host).pin_memory()
        return dict(kind=kind, trainer=trainer, tokens=tokens, targets=torch.roll(tokens, -1, dims=1).pin_memory())
    if kind == "logits":
        model = LlamaModel(_config(case), device="cuda", seed=seed)
        return dict(kind=kind, model=model,
                    tokens=torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=gen, device="cuda"))
    if kind == "attention":
        q, k, v = _qkv(case, gen, case["backward"])
        return dict(kind=kind, q=q, k=k, v=v, causal=case["causal"],
                    grad=_normal(gen, *q.shape) if case["backward"] else None)
    if kind == "sparse":
        q, k, v = _qkv(case, gen, True)
        module = SparseRingAttention(SparsePattern(window_tokens=case["window"], global_every=case["global_every"]),
                                     case["heads"], case["kv_heads"])
        return dict(kind=kind, module=module, q=q, k=k, v=v, grad=_normal(gen, *q.shape))
    if kind == "fp8kv":
        q, k, v = _qkv(case, gen, False)
        return dict(kind=kind, module=QuantizedRingAttention(case["heads"], case["kv_heads"]), q=q, k=k, v=v)
    M, K, N = case["rows"], case["inner"], case["outer"]
    return dict(kind=kind, x=_normal(gen, M, K).requires_grad_(True),
                w=_normal(gen, N, K, std=K ** -0.5).requires_grad_(True),
                residual=_normal(gen, M, N).requires_grad_(True), grad=_normal(gen, M, N))


def run(state):
    kind = state["kind"]
    if kind == "train":
        trainer = state["trainer"]
        loss = trainer.train_step(state["tokens"], state["targets"])
        opt = trainer.optimizer
        return dict(loss=loss, params=trainer.model.flat.params, m=opt.m, v=opt.v)
    if kind == "logits":
        return state["model"].logits(state["tokens"])
    if kind == "linear":
        leaves = (state["x"], state["w"], state["residual"])
        y = linear(*leaves)
        return (y.detach(), *torch.autograd.grad(y, leaves, state["grad"]))
    qkv = (state["q"], state["k"], state["v"])
    if kind == "attention":
        o = flash_attention(*qkv, causal=state["causal"])
        if state["grad"] is None:
            return o
    else:
        o = state["module"](*qkv)
        if kind == "fp8kv":
            return o
    return (o.detach(), *torch.autograd.grad(o, qkv, state["grad"]))


def _pairs(case):
    """Query-key pairs per head that the mask keeps (in whole 128 x 128 blocks above the diagonal's own)."""
    S = case["seq"]
    if case["kind"] == "sparse":
        pattern = SparsePattern(window_tokens=case["window"], global_every=case["global_every"])
        n = S // 128
        return pattern.density(S) * (n * (n + 1) // 2) * 128 * 128 - n * 128 * 127 // 2
    return S * (S + 1) // 2 if case.get("causal", True) else S * S


def work(case):
    kind = case["kind"]
    if kind in ("train", "logits"):
        cfg = _config(case)
        tokens = case["batch"] * case["seq"]
        per_token = cfg.flops_per_token(case["seq"])
        if kind == "train":   # weight, remainder and both moments read and written once; tokens and targets read
            return dict(bytes=24.0 * cfg.num_params() + 16.0 * tokens, flops=per_token * tokens)
        attn = 2.0 * case["seq"] * HEAD_DIM * cfg.n_heads * cfg.n_layers
        return dict(bytes=2.0 * cfg.num_params() + 2.0 * tokens * cfg.vocab_size,
                    flops=((per_token - 3.5 * attn) / 3 + attn) * tokens)
    if kind == "linear":
        M, K, N = case["rows"], case["inner"], case["outer"]   # y, dx and dw; x, w, residual and dy read, dy also returned
        return dict(bytes=2.0 * (2 * M * K + 2 * N * K + 3 * M * N), flops=6.0 * M * N * K)
    tokens = case.get("batch", 1) * case["seq"]
    q_bytes, kv_bytes = 2.0 * tokens * case["heads"] * HEAD_DIM, 2.0 * tokens * case["kv_heads"] * HEAD_DIM
    fwd = 4.0 * _pairs(case) * HEAD_DIM * case["heads"] * case.get("batch", 1)
    if kind == "fp8kv" or not case.get("backward", True):
        return dict(bytes=2 * q_bytes + 2 * kv_bytes, flops=fwd)
    return dict(bytes=4 * q_bytes + 4 * kv_bytes, flops=3.5 * fwd)   # q o dO dQ, k v dK dV


def tolerance(case):
    """About four times what this implementation differs by from the same path in fp64 (attention, linear) or in fp32
    on the host (the models): one attention 2.1e-3 to 2.5e-3 of the norm and up to 0.09 in one element (rows that see
    few keys have large gradients), one product 1.7e-3 and 4e-3 (the rounding to bf16), logits after two or three
    layers 5e-3 to 8e-3 and 0.05, gradients (the first moment) 6e-3 to 1e-2 and 0.34, second moments 1.1e-2."""
    return {"train": {"rel": 3e-2, "max": 0.99}, "logits": {"rel": 3e-2, "max": 0.2},
            "linear": {"rel": 7e-3, "max": 2e-2}}.get(case["kind"], {"rel": 1e-2, "max": 0.4})


# ------------------------------------------------------------------------------------------------
# The same passes in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------------


def _visible(case, row0, row1, device):
    """Indices of the keys that rows [row0, row1) may see, and which of them each row sees (None: all of them)."""
    S = case["seq"]
    if case["kind"] in ("train", "logits", "attention", "fp8kv"):
        if not case.get("causal", True):
            return torch.arange(S, device=device), None
        keys, window, every = torch.arange(row1, device=device), 0, 0
    else:
        window, every = case["window"] // 128, case["global_every"]
        keys = torch.arange(row1, device=device)
        keep = keys // 128 > row0 // 128 - window
        keys = keys[keep | (keys // 128 % every == 0)] if every else keys[keep]
    rows = torch.arange(row0, row1, device=device)[:, None]
    mask = keys[None] <= rows
    if window:
        near = rows // 128 - keys[None] // 128 < window
        mask &= (near | (keys[None] // 128 % every == 0)) if every else near
    return keys, mask


class _Attend64(torch.autograd.Function):
    """softmax(Q K^T / sqrt(d)) V, some rows of one KV head's query heads at a time."""

    @staticmethod
    def _pieces(case, q, k):
        B, S, Hq, _ = q.shape
        step = max(128, min(1024, 2 ** 28 // (S * (Hq // k.shape[2])) // 128 * 128))
        for r0 in range(0, S, step):
            r1 = min(S, r0 + step)
            keys, mask = _visible(case, r0, r1, q.device)
            for b in range(B):
                for h in range(k.shape[2]):
                    G = Hq // k.shape[2]
                    yield b, slice(r0, r1), slice(h * G, (h + 1) * G), h, keys, mask

    @staticmethod
    def _p(q, k, piece):
        b, rows, heads, h, keys, mask = piece
        s = q[b, rows, heads].transpose(0, 1) @ k[b, keys, h].T * HEAD_DIM ** -0.5     # [G, rows, keys]
        return torch.softmax(s if mask is None else s.masked_fill_(~mask, -math.inf), -1)

    @staticmethod
    def forward(ctx, q, k, v, case):
        o = torch.empty_like(q)
        for piece in _Attend64._pieces(case, q, k):
            b, rows, heads, h, keys, _ = piece
            o[b, rows, heads] = (_Attend64._p(q, k, piece) @ v[b, keys, h]).transpose(0, 1)
        ctx.save_for_backward(q, k, v)
        ctx.case = case
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v = ctx.saved_tensors
        dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for piece in _Attend64._pieces(ctx.case, q, k):
            b, rows, heads, h, keys, _ = piece
            p, g = _Attend64._p(q, k, piece), do[b, rows, heads].transpose(0, 1)
            dv[b, :, h].index_add_(0, keys, torch.einsum("grk,grd->kd", p, g))
            dp = g @ v[b, keys, h].T
            ds = p.mul_(dp - (dp * p).sum(-1, keepdim=True)).mul_(HEAD_DIM ** -0.5)
            dq[b, rows, heads] = (ds @ k[b, keys, h]).transpose(0, 1)
            dk[b, :, h].index_add_(0, keys, torch.einsum("grk,grd->kd", ds, q[b, rows, heads].transpose(0, 1)))
        return dq, dk, dv, None


def _hidden64(case, w, tokens):
    """The hidden states in front of the LM head; w: name -> weight in 64 bits."""
    cfg = _config(case)
    B, S = tokens.shape
    inv = cfg.rope_theta ** (-torch.arange(0, HEAD_DIM, 2, device="cuda", dtype=torch.float64) / HEAD_DIM)
    angle = torch.arange(S, device="cuda", dtype=torch.float64)[:, None] * inv
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def norm(x, weight):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.norm_eps) * weight

    def rotate(x):
        a, b = x.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    h = w["embed.weight"][tokens]
    for n in range(cfg.n_layers):
        p = "layers.%d." % n
        qkv = (norm(h, w[p + "norm1"]) @ w[p + "wqkv"].T).view(B, S, -1, HEAD_DIM)
        q, k, v = qkv.split([cfg.n_heads, cfg.n_kv_heads, cfg.n_kv_heads], 2)
        h = h + _Attend64.apply(rotate(q), rotate(k), v, case).reshape(B, S, -1) @ w[p + "wo"].T
        gate, up = (norm(h, w[p + "norm2"]) @ w[p + "wgu"].T).chunk(2, -1)
        h = h + (torch.nn.functional.silu(gate) * up) @ w[p + "wd"].T
    return norm(h, w["final_norm"])


def _exact_train(case, state):
    flat = state["trainer"].model.flat
    index, decay_end, total = dict(flat.index), flat.decay_end, flat.total
    params = flat.params.double()
    tokens, targets = state["tokens"].cuda(), state["targets"].cuda()
    state.clear()
    w = {n: params[o: o + math.prod(s)].view(s).requires_grad_(True) for n, (o, s) in index.items()}
    loss = torch.nn.functional.cross_entropy((_hidden64(case, w, tokens) @ w["lm_head.weight"].T).flatten(0, 1),
                                             targets.flatten())
    grads = torch.autograd.grad(loss, list(w.values()))
    g = torch.zeros(total, device="cuda", dtype=torch.float64)
    for (o, s), x in zip(index.values(), grads):
        g[o: o + math.prod(s)] = x.flatten()
    g *= min(1.0, 1.0 / (float(g.norm()) + 1e-6))
    params = params.detach()
    params[:decay_end] *= 1 - 3e-4 * 0.1
    return dict(loss=float(loss), params=params - 3e-4 * g / (g.abs() + 1e-8), m=0.1 * g, v=0.05 * g * g)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train" and work(case)["flops"] > 1.2e14:   # too long in 64 bits
        return None
    state = prepare(case, seed)
    if kind == "train":
        return _exact_train(case, state)
    if kind == "logits":
        flat = state["model"].flat
        w = {n: flat.param(n).double() for n in flat.index}
        with torch.no_grad():
            return _hidden64(case, w, state["tokens"]) @ w["lm_head.weight"].T
    wide = {n: x.detach().double() for n, x in state.items() if isinstance(x, torch.Tensor)}
    if kind == "linear":
        x, w, dy = wide["x"], wide["w"], wide["grad"]
        return x @ w.T + wide["residual"], dy @ w, dy.T @ x, dy
    if kind == "fp8kv":   # e4m3 codes with one 32-bit scale per head and 128 tokens are the format, not its error
        for n in "kv":
            x = state[n].float().unflatten(1, (-1, 128))
            scale = x.abs().amax((2, 4), keepdim=True) / 448
            wide[n] = ((x * (1 / scale)).to(torch.float8_e4m3fn).double() * scale.double()).flatten(1, 2)
    qkv = [wide[n].requires_grad_(True) for n in "qkv"]
    o = _Attend64.apply(*qkv, case)
    if kind == "fp8kv" or state["grad"] is None:
        return o.detach()
    return (o.detach(), *torch.autograd.grad(o, qkv, wide["grad"]))
