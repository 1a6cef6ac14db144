"""The work whose speed is tracked: one pass each of the training and inference paths of this package, through its
public entry points, on one GPU.

A case is a dict of plain values; ``kind`` says which path it takes:

    step    one optimizer step of the GPT trainer (forward, backward, clipping, AdamW) on tokens resident on the device
    block   one decoder block (attention + dense MLP), forward and backward or forward alone, bf16 or MXFP8 linears,
            optionally as a LoRA block over a frozen base
    moe     one mixture-of-experts decoder block (sink logits, optional sliding window), forward and backward
    flux    a cut of the MMDiT image model (one double block, two single blocks), training pass or sampling pass
    hstu    one HSTU layer over jagged user histories, forward and backward or forward alone
    embed   lookup of a batch's item ids in a large embedding table, and the sparse optimizer update of its gradient

``listed()`` are fixed sizes, ``draw(rng)`` gives others of the same ranges.
"""
import math
from statistics import NormalDist

import numpy as np
import torch

from mlperf_training_b200.models.gpt import Block, GPTConfig
from mlperf_training_b200.models.hstu import HSTUConfig, STULayer
from mlperf_training_b200.models.lora import freeze_base
from mlperf_training_b200.models.mmdit import MMDiT, MMDiTConfig
from mlperf_training_b200.ops.kernels import rope_tables
from mlperf_training_b200.parallel.embedding import ShardedEmbedding
from mlperf_training_b200.parallel.engine import OptimConfig
from mlperf_training_b200.trainer.pretrain import PretrainTrainer, TrainConfig

HEAD_DIM = 128
LR, BETA1, BETA2, ADAM_EPS, WEIGHT_DECAY, CLIP, WARMUP = 8e-4, 0.9, 0.95, 1e-5, 0.1, 1.0, 64
EMB_LR, EMB_EPS = 1e-2, 1e-8


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


# --------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest model of the smoke run: a step is a few hundred short launches
        dict(name="step_small", kind="step", layers=2, hidden=512, heads=4, kv=2, ffn=1024, vocab=2048, batch=2, seq=256,
             precision="bf16"),
        # the flagship: an 8B-parameter decoder's widths, vocabulary and sequence length, cut to one block
        dict(name="step_8b_layer", kind="step", layers=1, hidden=4096, heads=32, kv=8, ffn=14336, vocab=128256, batch=1,
             seq=8192, precision="mxfp8"),
        # fine-tuning on a batch of sequences that are no multiple of any tile, bf16 linears
        dict(name="block_ragged", kind="block", hidden=4096, heads=32, kv=8, ffn=14336, batch=3, seq=1337, precision="bf16",
             lora=0, train=True),
        # evaluation of the same block: forward alone, several sequences
        dict(name="block_eval", kind="block", hidden=4096, heads=32, kv=8, ffn=14336, batch=4, seq=2048, precision="mxfp8",
             lora=0, train=False),
        # adapter training of a 70B-parameter model's block over its frozen base, one sequence of 4096
        dict(name="lora_70b_layer", kind="block", hidden=8192, heads=64, kv=8, ffn=28672, batch=1, seq=4096, precision="bf16",
             lora=16, train=True),
        # mixture-of-experts pre-training, a sliding-window layer with block-scaled experts
        dict(name="moe_window", kind="moe", hidden=2880, heads=64, kv=8, ffn=2880, experts=32, top_k=4, batch=1, seq=8192, window=128,
             precision="mxfp8"),
        # the same model's full-attention layer in bf16 on a short batch
        dict(name="moe_full_short", kind="moe", hidden=2880, heads=64, kv=8, ffn=2880, experts=32, top_k=4, batch=1, seq=2000, window=0,
             precision="bf16"),
        # image-model training at the per-GPU micro-batch
        dict(name="flux_train", kind="flux", batch=8, precision="bf16", train=True),
        # sampling one image
        dict(name="flux_sample", kind="flux", batch=1, precision="bf16", train=False),
        # recommender training: a GPU's 128 users with log-normal history lengths
        dict(name="hstu_train", kind="hstu", users=128, median=512, train=True),
        # scoring a few users
        dict(name="hstu_score", kind="hstu", users=12, median=700, train=False),
        # item lookup and sparse update of about one GPU's batch
        dict(name="embed_update", kind="embed", ids=100000, rows=4000000, dim=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "block", "block", "block", "moe", "flux", "hstu", "hstu", "embed"])
    if kind == "step":
        heads = rng.choice([4, 8, 16])
        tokens = _log_int(rng, 256, 4096) // 8 * 8
        batch = rng.choice([1, 2, 4])
        return dict(kind=kind, layers=rng.choice([1, 2, 3]), hidden=heads * HEAD_DIM, heads=heads, kv=rng.choice([2, 4]),
                    ffn=heads * rng.choice([256, 384, 448]), vocab=rng.choice([2048, 8000, 32000]), batch=batch,
                    seq=max(tokens // batch, 16), precision=rng.choice(["bf16", "mxfp8"]))
    if kind == "block":
        heads = rng.choice([4, 8, 16, 32])
        batch = rng.choice([1, 1, 2, 3, 5])
        seq = max(_log_int(rng, 128, 8192) // batch, 32)
        precision = rng.choice(["bf16", "mxfp8"])
        if precision == "mxfp8":
            seq = (seq + 127) // 128 * 128
        return dict(kind=kind, hidden=heads * HEAD_DIM, heads=heads, kv=rng.choice([4, heads // 4 if heads >= 16 else 2]),
                    ffn=heads * 448, batch=batch, seq=seq, precision=precision,
                    lora=rng.choice([0, 0, 0, 16]), train=rng.random() < 0.7)
    if kind == "moe":
        return dict(kind=kind, hidden=2880, heads=64, kv=8, ffn=2880, experts=32, top_k=4, batch=1, seq=_log_int(rng, 300, 8192),
                    window=rng.choice([0, 128]), precision=rng.choice(["bf16", "mxfp8"]))
    if kind == "flux":
        return dict(kind=kind, batch=rng.randint(1, 8), precision="bf16", train=rng.random() < 0.6)
    if kind == "hstu":
        return dict(kind=kind, users=_log_int(rng, 4, 128), median=_log_int(rng, 100, 512), train=rng.random() < 0.6)
    return dict(kind="embed", ids=_log_int(rng, 3000, 200000), rows=_log_int(rng, 100000, 4000000), dim=256)


# --------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=_dev()).manual_seed(1000003 * int(seed) + 17)


def _normal(g, shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=g, device=_dev(), dtype=torch.float32) * std).to(dtype)


def _fill(named, g, std):
    """Weights of a module from the seed: matrices normal (those that write to the residual stream of a decoder at the
    1 / 8 of a 32-layer initialisation, its token embedding at the size of a trained residual stream), norm weights about
    one, biases and sinks about zero."""
    with torch.no_grad():
        for name, p in named:
            if p.dim() >= 2:
                s = std
                if name.endswith(("lora_qkv.a", "lora_proj.a")):
                    s = p.shape[1] ** -0.5
                elif name.endswith(("w_proj", "mlp.w_down", "mlp.w2")):
                    s = std / 8
                elif name == "embed":
                    s = 0.5
                p.copy_(torch.randn(p.shape, generator=g, device=p.device, dtype=torch.float32) * s)
            elif "norm_b" in name or "bias" in name or "beta" in name or "sink" in name:
                p.copy_(torch.randn(p.shape, generator=g, device=p.device, dtype=torch.float32) * 0.1)
            else:
                p.copy_(1.0 + torch.randn(p.shape, generator=g, device=p.device, dtype=torch.float32) * 0.1)


def _gpt_config(c):
    moe = c["kind"] == "moe"
    over = dict(n_experts=c["experts"], top_k=c["top_k"], moe_ffn_hidden=c["ffn"], sink=True, window=c["window"], head_dim=64,
                window_layers="even" if c["window"] else "none", rope_theta=150000.0, norm_eps=1e-6) if moe else {}
    if c.get("lora"):
        over.update(lora_rank=c["lora"], lora_alpha=32.0, lora_dropout=0.0)
    base = dict(name=c["kind"], n_layers=c.get("layers", 1), hidden=c["hidden"], n_heads=c["heads"], n_kv_heads=c["kv"],
                head_dim=HEAD_DIM, ffn_hidden=c["ffn"], vocab_size=c.get("vocab", 2048), seq_len=c["seq"], rope_theta=500000.0,
                precision=c["precision"])
    base.update(over)
    return GPTConfig(**base)


def _step_inputs(c, seed):
    g = _gen(seed)
    tokens = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=g, device=_dev(), dtype=torch.int64)
    return g, tokens


def _block(c, seed):
    """(block, x, gradient of the output): rows of the residual stream and of its gradient."""
    cfg = _gpt_config(c)
    blk = Block(cfg, 0, torch.bfloat16, _dev())
    g = _gen(seed)
    _fill(blk.named_parameters(), g, 0.02)
    if c.get("lora"):
        freeze_base(blk)
    T = c["batch"] * c["seq"]
    x = _normal(g, (T, c["hidden"]))
    dy = _normal(g, (T, c["hidden"]), 0.01)
    if c["kind"] == "moe":
        # a trained router tells its experts apart: every token leans towards top_k of them, some experts more wanted than others
        want = torch.rand((T, c["experts"]), generator=g, device=_dev()) ** torch.linspace(0.7, 1.4, c["experts"], device=_dev())
        pick = torch.zeros_like(want).scatter_(1, want.topk(c["top_k"], 1).indices, 1.0)
        rows = torch.nn.functional.normalize(blk.mlp.router.detach().float(), dim=1)
        x = (x.float() + 6.0 * (pick @ rows)).to(x.dtype)
    return cfg, blk, x, dy


def _flux(c, seed):
    cfg = MMDiTConfig(name="mmdit-cut", n_double=1, n_single=2, precision=c["precision"])
    model = MMDiT(cfg, _dev(), seed=0)
    g = _gen(seed)
    _fill(model.named_parameters(), g, 0.02)
    B = c["batch"]
    img = _normal(g, (B, cfg.img_tokens, cfg.in_channels))
    txt = _normal(g, (B, cfg.txt_tokens, cfg.txt_dim))
    vec = _normal(g, (B, cfg.vec_dim))
    t = torch.rand((B,), generator=g, device=_dev())
    target = _normal(g, (B, cfg.img_tokens, cfg.in_channels), dtype=torch.float32)
    return cfg, model, (img, txt, vec, t, target)


def _lengths(c):
    """History lengths of the batch: the quantiles of a log-normal (sigma 1), cut to [16, 4096]."""
    nd, n = NormalDist(), c["users"]
    return [int(min(max(c["median"] * math.exp(nd.inv_cdf((i + 0.5) / n)), 16), 4096)) for i in range(n)]


def _hstu(c, seed):
    cfg = HSTUConfig(layers=1, dim=512, heads=4, d_qk=128, d_v=128, max_seq_len=4096, linear_dropout=0.0, dtype="bf16")
    layer = STULayer(cfg, torch.bfloat16, _dev())
    g = _gen(seed)
    _fill(layer.named_parameters(), g, 0.04)
    lengths = np.array(_lengths(c))[np.random.RandomState(int(seed) % (2 ** 31)).permutation(c["users"])]
    offsets = torch.tensor(np.concatenate([[0], np.cumsum(lengths)]), dtype=torch.int32, device=_dev())
    targets = torch.ones(c["users"], dtype=torch.int32, device=_dev())
    n = int(lengths.sum())
    rows = (n + 127) // 128 * 128
    x, dy = _normal(g, (rows, cfg.dim)), _normal(g, (rows, cfg.dim), 0.01)
    x[n:] = 0
    dy[n:] = 0
    layer.train(bool(c["train"]))
    return cfg, layer, lengths, offsets, targets, rows, x, dy


def _embed_inputs(c, seed):
    """Zipf-distributed ids (exponent about 1.05 over the table), gradient rows."""
    g = _gen(seed)
    u = torch.rand((c["ids"],), generator=g, device=_dev(), dtype=torch.float64)
    a = 0.05                                         # inverse of the continuous Zipf distribution function
    top = float(c["rows"]) ** -a
    rank = (1.0 - u * (1.0 - top)) ** (-1.0 / a)
    ids = (rank.long().clamp(1, c["rows"]) * 2654435761) % c["rows"]
    return ids, _normal(g, (c["ids"], c["dim"]), 0.1)


def prepare(case, seed):
    c = case
    if c["kind"] == "step":
        cfg = _gpt_config(c)
        opt = OptimConfig(lr=LR, beta1=BETA1, beta2=BETA2, eps=ADAM_EPS, weight_decay=WEIGHT_DECAY, clip_grad=CLIP)
        tr = PretrainTrainer(cfg, opt, TrainConfig(micro_batch=c["batch"], local_batch=c["batch"], warmup_steps=WARMUP), _dev())
        g, tokens = _step_inputs(c, seed)
        _fill(tr.model.named_parameters(), g, 0.02)
        moments = {n: b.m[o:o + p.numel()] for b in tr.engine.buckets for (n, p), o in zip(b.params, b.offsets)}
        return dict(case=c, trainer=tr, tokens=tokens, moments=moments)
    if c["kind"] in ("block", "moe"):
        cfg, blk, x, dy = _block(c, seed)
        cos, sin = rope_tables(c["seq"], cfg.head_dim, cfg.rope_theta, _dev())
        names = [n for n, p in blk.named_parameters() if p.requires_grad]
        return dict(case=c, block=blk, x=x.requires_grad_(bool(c.get("train", True))), dy=dy, cos=cos, sin=sin, names=names)
    if c["kind"] == "flux":
        cfg, model, inputs = _flux(c, seed)
        return dict(case=c, model=model, inputs=inputs, names=[n for n, _ in model.named_parameters()])
    if c["kind"] == "hstu":
        cfg, layer, _, offsets, targets, rows, x, dy = _hstu(c, seed)
        return dict(case=c, layer=layer, offsets=offsets, targets=targets, rows=rows, dy=dy, x=x.requires_grad_(bool(c["train"])),
                    names=[n for n, _ in layer.named_parameters()])
    ids, dy = _embed_inputs(c, seed)
    table = ShardedEmbedding(c["rows"], c["dim"], device=_dev(), lr=EMB_LR, eps=EMB_EPS, seed=int(seed) % 1000)
    return dict(case=c, table=table, ids=ids, dy=dy)


# --------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------
def _grads(y, dy, x, module, names):
    params = dict(module.named_parameters())
    got = torch.autograd.grad(y, [x] + [params[n] for n in names], dy)
    return {"y": y.detach(), "dx": got[0], "grads": dict(zip(names, got[1:]))}


def run(state):
    c = state["case"]
    if c["kind"] == "step":
        tr = state["trainer"]
        loss = tr.train_step_device(state["tokens"])
        return {"loss": loss, "weights": {n: p.detach() for n, p in tr.model.named_parameters()}, "moments": state["moments"]}
    if c["kind"] in ("block", "moe"):
        args = (state["cos"], state["sin"], c["batch"], c["seq"])
        if not c.get("train", True):
            with torch.no_grad():
                return state["block"](state["x"], *args)
        return _grads(state["block"](state["x"], *args), state["dy"], state["x"], state["block"], state["names"])
    if c["kind"] == "flux":
        img, txt, vec, t, target = state["inputs"]
        if not c["train"]:
            with torch.no_grad():
                return state["model"](img, txt, vec, t)
        pred = state["model"](img, txt, vec, t)
        loss = ((pred.float() - target) ** 2).mean()
        params = dict(state["model"].named_parameters())
        got = torch.autograd.grad(loss, [params[n] for n in state["names"]])
        return {"loss": loss.detach(), "pred": pred.detach(), "grads": _stack_small(dict(zip(state["names"], got)))}
    if c["kind"] == "hstu":
        if not c["train"]:
            with torch.no_grad():
                return state["layer"](state["x"], state["offsets"], state["targets"], state["rows"])
        y = state["layer"](state["x"], state["offsets"], state["targets"], state["rows"])
        return _grads(y, state["dy"], state["x"], state["layer"], state["names"])
    table = state["table"]
    out = table.lookup(state["ids"])
    out.backward(state["dy"])
    return {"rows": out.detach(), "weight": table.weight, "sums": table.state}


def _stack_small(grads):
    """The vectors among the gradients as one list per width, the matrices by name (a model has many small biases)."""
    small = {}
    for n, g in grads.items():
        if g.dim() == 1:
            small.setdefault("width%d" % g.numel(), []).append(g)
    out = {n: g for n, g in grads.items() if g.dim() > 1}
    out.update({k: torch.stack(v) for k, v in small.items()})
    return out


# --------------------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------------------
def _pairs(S, window, causal=True):
    """Query-key pairs one head of one sequence looks at."""
    if not causal:
        return S * S
    if window and window < S:
        return window * S - window * (window - 1) // 2
    return S * (S + 1) // 2


def work(case):
    c = case
    if c["kind"] in ("step", "block", "moe"):
        hd = 64 if c["kind"] == "moe" else HEAD_DIM
        d, T = c["hidden"], c["batch"] * c["seq"]
        attn_w = d * (c["heads"] + 2 * c["kv"]) * hd + c["heads"] * hd * d
        attn = 4 * c["heads"] * hd * c["batch"] * _pairs(c["seq"], c.get("window", 0))
        if c["kind"] == "moe":
            held, used = attn_w + c["experts"] * 3 * d * c["ffn"], attn_w + c["top_k"] * 3 * d * c["ffn"] + c["experts"] * d
        else:
            held = used = attn_w + 3 * d * c["ffn"]
        if c["kind"] == "step":
            n = c["layers"] * held + 2 * c["vocab"] * d
            flops = 6 * T * (c["layers"] * used + c["vocab"] * d) + c["layers"] * 3.5 * attn
            # weights read and written in bf16, both moments read and written in fp32, tokens read
            return {"bytes": n * (2 + 2 + 16) + 8 * T, "flops": flops}
        if not c.get("train", True):
            return {"bytes": 2 * held + 4 * T * d, "flops": 2 * T * used + attn}
        if c.get("lora"):
            return {"bytes": 2 * held + 8 * T * d, "flops": 4 * T * used + 3.5 * attn}
        return {"bytes": 4 * held + 8 * T * d, "flops": 6 * T * used + 3.5 * attn}
    if c["kind"] == "flux":
        cfg = MMDiTConfig(n_double=1, n_single=2)
        d, m, B, S = cfg.hidden, cfg.mlp_hidden, c["batch"], cfg.img_tokens + cfg.txt_tokens
        double, single = 4 * d * d + 2 * d * m, 3 * d * d + d * m + (d + m) * d
        ends = cfg.txt_dim * d + 2 * cfg.in_channels * d
        mods = 12 * d * d + 2 * 3 * d * d + 2 * d * d + (256 + cfg.vec_dim + 2 * d) * d
        held = 2 * double + 2 * single + ends + mods
        gemm = 2 * B * S * (double + 2 * single) + 2 * B * (cfg.txt_tokens * cfg.txt_dim + 2 * cfg.img_tokens * cfg.in_channels) * d + 2 * B * mods
        attn = 3 * 4 * B * S * S * d
        io = 2 * B * (2 * cfg.img_tokens * cfg.in_channels + cfg.txt_tokens * cfg.txt_dim)
        if c["train"]:
            return {"bytes": 4 * held + io, "flops": 3 * gemm + 3.5 * attn}
        return {"bytes": 2 * held + io, "flops": gemm + attn}
    if c["kind"] == "hstu":
        lens, d = _lengths(c), 512
        T, pairs = sum(lens), sum(n * (n + 1) // 2 for n in lens)
        gemm, attn = 2 * T * (d * 2048 + 1536 * d), 4 * 512 * pairs
        if c["train"]:
            return {"bytes": 4 * 7 * d * d + 8 * T * d, "flops": 3 * gemm + 3.5 * attn}
        return {"bytes": 2 * 7 * d * d + 4 * T * d, "flops": gemm + attn}
    # ids, output rows and gradient rows once; each of (at most) n table rows and sums read and written
    n, d = c["ids"], c["dim"]
    uniq = n // 2
    return {"bytes": 8 * n + 4 * n * d + uniq * (4 * d + 8), "flops": 4 * n * d}


def tolerance(case):
    """bf16 activations between the operators (8 mantissa bits) set the difference of two correct implementations; with
    block-scaled linears a last-bit change of an activation can move its 8-bit code by a step."""
    if case["kind"] == "embed":
        return {"rel": 1e-3, "max": 0.05}
    if case.get("precision") == "mxfp8":
        return {"rel": 0.03, "max": 0.9}
    return {"rel": 0.015, "max": 0.6}


# --------------------------------------------------------------------------------------
# the same passes in 64 bits, in plain torch
# --------------------------------------------------------------------------------------
def _ck(fn, *args):
    from torch.utils.checkpoint import checkpoint
    return checkpoint(fn, *args, use_reentrant=False) if torch.is_grad_enabled() else fn(*args)


def _rms(x, w, eps):
    n = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return n if w is None else n * w


def _ln(x, w=None, b=None, eps=1e-6):
    n = (x - x.mean(-1, keepdim=True)) * torch.rsqrt(x.var(-1, unbiased=False, keepdim=True) + eps)
    return n if w is None else n * w + b


def _rotate(x, cos, sin):
    """x [..., S, H, D], tables [S, D / 2], rotate-half."""
    h = x.shape[-1] // 2
    a, b = x[..., :h], x[..., h:]
    c, s = cos[:, None, :], sin[:, None, :]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _one_head(q, k, v, ok, scale, sink):
    s = (q @ k.t()) * scale
    if ok is not None:
        s = s.masked_fill(~ok, float("-inf"))
    if sink is None:
        return torch.softmax(s, -1) @ v
    p = torch.softmax(torch.cat([s, sink.reshape(1, 1).expand(s.shape[0], 1)], 1), -1)
    return p[:, :-1] @ v


def _attend(q, k, v, causal, window=0, sink=None):
    """[B, S, H, D] tensors in 64 bits; one head at a time, recomputed in backward."""
    B, S, H, D = q.shape
    g, ok = H // k.shape[2], None
    if causal:
        i = torch.arange(S, device=q.device)
        ok = i[:, None] >= i[None, :]
        if window:
            ok &= (i[:, None] - i[None, :]) < window
    outs = []
    for b in range(B):
        heads = [_ck(_one_head, q[b, :, h], k[b, :, h // g], v[b, :, h // g], ok, D ** -0.5, None if sink is None else sink[h])
                 for h in range(H)]
        outs.append(torch.stack(heads, 1))
    return torch.stack(outs, 0)


def _mlp(h, wn, wgu, wd, eps):
    gate, up = (_rms(h, wn, eps) @ wgu.t()).chunk(2, -1)
    return h + (torch.nn.functional.silu(gate) * up) @ wd.t()


def _experts(h, p, c, eps):
    hn = _rms(h, p["mlp_norm"], eps)
    logits = hn @ p["mlp.router"].t()
    val, idx = torch.topk(logits, c["top_k"], -1)
    w = torch.softmax(val, -1)
    out = h
    for e in range(c["experts"]):
        t, slot = torch.nonzero(idx == e, as_tuple=True)
        gate, up = (hn[t] @ p["mlp.w1"][e].t()).chunk(2, -1)
        y = (torch.nn.functional.silu(gate) * up) @ p["mlp.w2"][e].t()
        out = out.index_add(0, t, y * w[t, slot][:, None])
    return out


def _exact_block(x, p, c, cfg, cos, sin):
    B, S, H, G, D, eps = c["batch"], c["seq"], c["heads"], c["kv"], cfg.head_dim, cfg.norm_eps
    xn = _rms(x, p["attn_norm"], eps)
    qkv = xn @ p["w_qkv"].t()
    scale = 32.0 / c["lora"] if c.get("lora") else 0.0
    if c.get("lora"):
        qkv = qkv + scale * (xn @ p["lora_qkv.a"].t()) @ p["lora_qkv.b"].t()
    qkv = qkv.view(B, S, -1, D)
    q, k, v = _rotate(qkv[:, :, :H], cos, sin), _rotate(qkv[:, :, H:H + G], cos, sin), qkv[:, :, H + G:]
    a = _attend(q, k, v, True, c.get("window", 0), p.get("sink")).reshape(B * S, H * D)
    h = x + a @ p["w_proj"].t()
    if c.get("lora"):
        h = h + scale * (a @ p["lora_proj.a"].t()) @ p["lora_proj.b"].t()
    if c["kind"] == "moe":
        return _experts(h, p, c, eps)
    return _ck(_mlp, h, p["mlp_norm"], p["mlp.w_gate_up"], p["mlp.w_down"], eps)


def _double(named, grad):
    return {n: p.detach().double().requires_grad_(grad and p.requires_grad) for n, p in named}


def _tables(c, cfg):
    cos, sin = rope_tables(c["seq"], cfg.head_dim, cfg.rope_theta, _dev())
    return cos.double(), sin.double()


def _exact_grads(y, dy, x, p, names):
    got = torch.autograd.grad(y, [x] + [p[n] for n in names], dy.double())
    return {"y": y.detach(), "dx": got[0], "grads": dict(zip(names, got[1:]))}


def _exact_step(c, seed):
    state = prepare(c, seed)
    cfg, named = state["trainer"].cfg, [(n, p.detach().clone()) for n, p in state["trainer"].model.named_parameters()]
    tokens = state["tokens"]
    state = None
    p = {n: t.double().requires_grad_(True) for n, t in named}
    cos, sin = _tables(c, cfg)
    x = p["embed"][tokens[:, :-1].reshape(-1)]
    for i in range(c["layers"]):
        pre = "blocks.%d." % i
        x = _exact_block(x, {n[len(pre):]: t for n, t in p.items() if n.startswith(pre)}, c, cfg, cos, sin)
    labels = tokens[:, 1:].reshape(-1)

    def head(x, wn, w, lab):
        return torch.nn.functional.cross_entropy(_rms(x, wn, cfg.norm_eps) @ w.t(), lab, reduction="sum")
    total = sum(_ck(head, x[i:i + 2048], p["final_norm"], p["lm_head"], labels[i:i + 2048]) for i in range(0, len(x), 2048))
    loss = total / labels.numel()
    names = list(p)
    grads = dict(zip(names, torch.autograd.grad(loss, [p[n] for n in names])))
    norm = math.sqrt(sum(float((g * g).sum()) for g in grads.values()))
    coef = min(1.0, CLIP / (norm + 1e-6))
    lr = LR / WARMUP
    weights, moments = {}, {}
    for n in names:
        g, w = grads.pop(n) * coef, p.pop(n).detach()
        decay = WEIGHT_DECAY if (w.dim() >= 2 and "norm" not in n) else 0.0
        moments[n] = ((1 - BETA1) * g).reshape(-1)
        weights[n] = w * (1 - lr * decay) - lr * g / (g.abs() + ADAM_EPS)
    # 8-bit copies of d(loss)/d(logits) drop the softmax's tail beside the label's entry of the same scale block: the gradients
    # of that recipe are 0.07 to 0.17 from these and say nothing about the arithmetic around them
    return {"loss": loss.detach(), "weights": weights, "moments": moments if c["precision"] == "bf16" else dict.fromkeys(moments)}


def _exact_flux(c, seed):
    cfg, model, (img, txt, vec, t, target) = _flux(c, seed)
    p = _double(model.named_parameters(), c["train"])
    cos, sin = (z.double() for z in model.rope(torch.device(_dev())))
    B, H, D, d = c["batch"], cfg.n_heads, cfg.head_dim, cfg.hidden
    silu = torch.nn.functional.silu

    def lin(x, n):
        return x @ p[n + ".weight"].t() + p[n + ".bias"]

    def gelu(x):
        return torch.nn.functional.gelu(x, approximate="tanh")

    def mod(x, shift, scale):
        return _ln(x) * (1 + scale[:, None]) + shift[:, None]

    half = 128
    freqs = torch.exp(-math.log(10000.0) * torch.arange(half, dtype=torch.float64, device=t.device) / half)
    arg = (t.double() * 1000.0)[:, None] * freqs[None]
    temb = torch.cat([arg.cos(), arg.sin()], -1)
    v = silu(lin(silu(lin(temb, "time_in1")), "time_in2") + lin(silu(lin(vec.double(), "vec_in1")), "vec_in2"))
    x = {"img": lin(img.double(), "img_in"), "txt": lin(txt.double(), "txt_in")}
    St = cfg.txt_tokens
    parts = {}
    b = "double_blocks.0."
    for s in ("img", "txt"):
        m = lin(v, b + s + "_mod").chunk(6, -1)
        qkv = lin(mod(x[s], m[0], m[1]), b + s + "_qkv").view(B, -1, 3, H, D)
        parts[s] = (_rms(qkv[:, :, 0], p[b + s + "_qknorm.q_scale"], 1e-6), _rms(qkv[:, :, 1], p[b + s + "_qknorm.k_scale"], 1e-6),
                    qkv[:, :, 2], m)
    q, k, val = (torch.cat([parts["txt"][i], parts["img"][i]], 1) for i in range(3))
    a = _attend(_rotate(q, cos, sin), _rotate(k, cos, sin), val, False).reshape(B, -1, d)
    for s, part in (("txt", a[:, :St]), ("img", a[:, St:])):
        m = parts[s][3]
        h = x[s] + lin(part, b + s + "_proj") * m[2][:, None]
        x[s] = h + lin(gelu(lin(mod(h, m[3], m[4]), b + s + "_fc1")), b + s + "_fc2") * m[5][:, None]
    y = torch.cat([x["txt"], x["img"]], 1)
    for i in range(cfg.n_single):
        b = "single_blocks.%d." % i
        shift, scale, gate = lin(v, b + "mod").chunk(3, -1)
        z = lin(mod(y, shift, scale), b + "linear1")
        qkv = z[..., :3 * d].reshape(B, -1, 3, H, D)
        q, k = _rms(qkv[:, :, 0], p[b + "qknorm.q_scale"], 1e-6), _rms(qkv[:, :, 1], p[b + "qknorm.k_scale"], 1e-6)
        a = _attend(_rotate(q, cos, sin), _rotate(k, cos, sin), qkv[:, :, 2], False).reshape(B, -1, d)
        y = y + lin(torch.cat([a, gelu(z[..., 3 * d:])], -1), b + "linear2") * gate[:, None]
    shift, scale = lin(v, "final_mod").chunk(2, -1)
    pred = lin(mod(y[:, St:], shift, scale), "final_out")
    if not c["train"]:
        return pred.detach()
    loss = ((pred - target.double()) ** 2).mean()
    names = list(p)
    got = torch.autograd.grad(loss, [p[n] for n in names])
    return {"loss": loss.detach(), "pred": pred.detach(), "grads": _stack_small(dict(zip(names, got)))}


def _exact_hstu(c, seed):
    cfg, layer, lengths, offsets, _, rows, x, dy = _hstu(c, seed)
    p = _double(layer.named_parameters(), c["train"])
    x = x.double().requires_grad_(bool(c["train"]))
    h, D = cfg.heads, 128
    uvqk = _ln(x, p["in_norm_w"], p["in_norm_b"]) @ p["uvqk_weight"].t() + p["uvqk_beta"]
    u, v, q, k = uvqk.split([h * D] * 4, 1)

    def user(q, k, v):
        n = len(q)
        i = torch.arange(n, device=q.device)
        ids = i.clamp(max=n - 1)                   # one target: the last position
        ok = (i[:, None] == i[None, :]) | (ids[:, None] > ids[None, :])
        q, k, v = (t.view(n, h, D).transpose(0, 1) for t in (q, k, v))
        s = torch.nn.functional.silu(q @ k.transpose(1, 2) * D ** -0.5) / cfg.attn_len()
        return ((s * ok) @ v).transpose(0, 1).reshape(n, h * D)
    outs, at = [], 0
    for n in lengths:
        outs.append(_ck(user, q[at:at + n], k[at:at + n], v[at:at + n]))
        at += int(n)
    outs.append(torch.zeros(rows - at, h * D, dtype=torch.float64, device=x.device))
    a, u = torch.cat(outs), torch.nn.functional.silu(u)
    y = x + torch.cat([u, a, u * _ln(a, p["out_norm_w"], p["out_norm_b"])], 1) @ p["out_weight"].t()
    if not c["train"]:
        return y.detach()
    return _exact_grads(y, dy, x, p, list(p))


def _exact_embed(c, seed):
    state = prepare(c, seed)
    w, ids, dy = state["table"].weight.double(), state["ids"], state["dy"].double()
    out = w[ids]
    uniq, inv = torch.unique(ids, return_inverse=True)
    g = torch.zeros(len(uniq), c["dim"], dtype=torch.float64, device=w.device).index_add_(0, inv, dy)
    sums = torch.zeros(c["rows"], dtype=torch.float64, device=w.device)
    sums[uniq] = (g * g).mean(-1)
    w[uniq] -= EMB_LR * g / (sums[uniq].sqrt()[:, None] + EMB_EPS)
    return {"rows": out, "weight": w, "sums": sums}


def exact(case, seed):
    c = case
    if c["kind"] == "step":
        return _exact_step(c, seed)
    if c["kind"] in ("block", "moe"):
        cfg, blk, x, dy = _block(c, seed)
        train = bool(c.get("train", True))
        p = _double(blk.named_parameters(), train)
        names = [n for n, t in blk.named_parameters() if t.requires_grad]
        blk = None
        x = x.double().requires_grad_(train)
        y = _exact_block(x, p, c, cfg, *_tables(c, cfg))
        return _exact_grads(y, dy, x, p, names) if train else y.detach()
    if c["kind"] == "flux":
        return _exact_flux(c, seed)
    if c["kind"] == "hstu":
        return _exact_hstu(c, seed)
    return _exact_embed(c, seed)
