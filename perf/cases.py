"""Performance cases of the framework: what its users have it do on one GPU, through its public entry points.

Seven kinds of work:

  llama      one optimizer step of a Llama-shaped pipeline (``build_llama_pipeline`` / ``train_step``)
  gpt2       one optimizer step of a GPT-2-shaped pipeline (``build_gpt2_pipeline`` / ``train_step``)
  score      forward only: logits and mean loss of a batch of prompts (``Llama`` under ``no_grad``)
  attention  rotary + causal attention, forward and backward (``rope_attention``)
  head       LM-head projection and cross-entropy, forward and backward (``linear`` + the families' losses)
  moe        routed expert layer, forward and backward (``MoEFeedForward``)
  adamw      fused optimizer update alone (``FusedAdamW.step``)

Model widths are those of the families' own configurations (Llama-2-7B and -13B, GPT-2 small, the 8-expert top-2 MoE);
depths are cut so that the weights, moments and activations of several states fit one GPU.
"""
import math
import random

import torch
import torch.utils.checkpoint

from pippy_b200.models.gpt2 import GPT2Config, gpt2_loss
from pippy_b200.models.llama import Llama, LlamaConfig, causal_lm_loss
from pippy_b200.ops import functional as pf
from pippy_b200.optim import FlatParams, FusedAdamW
from pippy_b200.parallel.ep import EPContext, MoEFeedForward
from pippy_b200.train import build_gpt2_pipeline, build_llama_pipeline

BF16 = torch.bfloat16


def listed():
    return [
        # the smallest training job: four narrow layers, two stages on the GPU; nearly all of it is launches
        dict(name="train_llama_tiny", kind="llama", dim=512, layers=4, heads=4, kv_heads=4, ffn=1024, vocab=1024, batch=4,
             seq=256, microbatches=2, schedule="interleaved_1f1b", stages=2, checkpoint=False),
        # GPT-2 small, one data-parallel replica's share of the 64 x 1024 batch: 16 microbatches of 2 x 1024 tokens
        dict(name="train_gpt2_small", kind="gpt2", dim=768, layers=12, heads=12, vocab=50257, batch=32, seq=1024,
             microbatches=16, schedule="1f1b"),
        # Llama-2-7B width with the benchmark's microbatch of 2 x 4096 tokens and two stages per rank
        dict(name="train_llama_7b_width", kind="llama", dim=4096, layers=2, heads=32, kv_heads=32, ffn=11008, vocab=32000,
             batch=4, seq=4096, microbatches=2, schedule="interleaved_1f1b", stages=2, checkpoint=False),
        # Llama-2-13B width, zero-bubble (split backward), activation checkpointing, a sequence that fills no tile
        dict(name="train_llama_13b_ragged", kind="llama", dim=5120, layers=2, heads=40, kv_heads=40, ffn=13824,
             vocab=32000, batch=2, seq=2999, microbatches=2, schedule="zero_bubble", stages=1, checkpoint=True),
        # scoring one short prompt: the weights are read once for 77 tokens
        dict(name="score_short", kind="score", dim=4096, layers=4, heads=32, kv_heads=32, ffn=11008, vocab=32000, batch=1,
             seq=77),
        # scoring a batch of medium prompts with grouped-query attention
        dict(name="score_batch_gqa", kind="score", dim=4096, layers=4, heads=32, kv_heads=8, ffn=14336, vocab=32000,
             batch=3, seq=1365),
        # GPT-2 small's attention on one microbatch: head size 64, no rotary
        dict(name="attention_gpt2", kind="attention", batch=2, seq=1024, heads=12, kv_heads=12, head_dim=64, rotary=False),
        # the benchmark microbatch's attention: 2 x 4096 tokens, 32 heads of 128
        dict(name="attention_7b", kind="attention", batch=2, seq=4096, heads=32, kv_heads=32, head_dim=128, rotary=True),
        # long context with grouped-query heads, as in the MoE family
        dict(name="attention_long_gqa", kind="attention", batch=1, seq=16384, heads=32, kv_heads=8, head_dim=128,
             rotary=True),
        # GPT-2's 50257-way head on one microbatch (padded vocabulary, tied-width 768)
        dict(name="head_gpt2", kind="head", family="gpt2", tokens=2048, dim=768, vocab=50257),
        # one expert layer: 8 experts, top-2, one sequence of 4096 tokens
        dict(name="moe_layer", kind="moe", tokens=4096, dim=4096, ffn=14336, experts=8, top_k=2),
        # the update of a GPT-2-sized stage with fp32 master weights; a parameter count that is no multiple of anything
        dict(name="adamw_master", kind="adamw", numel=124439807, master=True),
    ]


def _between(rng, lo, hi):
    """An integer from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["llama", "llama", "gpt2", "score", "score", "attention", "attention", "head", "moe", "adamw"])
    if kind in ("llama", "score"):
        hd = rng.choice([64, 128, 128])
        heads = _between(rng, 4, 40 if hd == 128 else 16)
        kv = heads // 4 if heads % 4 == 0 and rng.random() < 0.4 else heads
        dim = heads * hd
        case = dict(kind=kind, dim=dim, layers=rng.randint(2, 4), heads=heads, kv_heads=kv,
                    ffn=8 * int(dim * rng.uniform(2.0, 3.5) / 8), vocab=8 * _between(rng, 64, 4000))
        if kind == "llama":
            mbs = rng.randint(2, 4)
            schedule = rng.choice(["1f1b", "interleaved_1f1b", "zero_bubble"])
            case.update(batch=mbs * rng.randint(1, 3), seq=_between(rng, 64, 4096), microbatches=mbs, schedule=schedule,
                        stages=2 if schedule == "interleaved_1f1b" else 1, checkpoint=rng.random() < 0.25)
        else:
            case.update(batch=rng.randint(1, 4), seq=_between(rng, 16, 4096))
    elif kind == "gpt2":
        heads = rng.randint(4, 12)
        mbs = rng.randint(2, 12)
        case = dict(kind=kind, dim=64 * heads, layers=rng.randint(4, 12), heads=heads, vocab=_between(rng, 500, 50257),
                    batch=mbs * rng.randint(1, 2), seq=_between(rng, 64, 1024), microbatches=mbs,
                    schedule=rng.choice(["1f1b", "gpipe"]))
    elif kind == "attention":
        hd = rng.choice([64, 128, 128])
        heads = _between(rng, 4, 32)
        kv = heads // 4 if heads % 4 == 0 and rng.random() < 0.5 else heads
        case = dict(kind=kind, batch=rng.randint(1, 4), seq=_between(rng, 64, 12000), heads=heads, kv_heads=kv,
                    head_dim=hd, rotary=rng.random() < 0.7)
    elif kind == "head":
        case = dict(kind=kind, family=rng.choice(["gpt2", "llama"]), tokens=_between(rng, 128, 8192),
                    dim=64 * rng.randint(4, 64), vocab=8 * _between(rng, 128, 6300))
    elif kind == "moe":
        case = dict(kind=kind, tokens=_between(rng, 128, 4096), dim=128 * rng.randint(2, 32),
                    ffn=128 * _between(rng, 4, 112), experts=rng.choice([4, 8]), top_k=2)
    else:
        case = dict(kind=kind, numel=_between(rng, 100_000, 400_000_000), master=rng.random() < 0.5)
    while work(case)["flops"] > 3.0e13:  # no dearer than the listed ones
        case["seq"] = max(16, int(case["seq"] * 0.7))
    return case


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _llama_config(c):
    return LlamaConfig(vocab_size=c["vocab"], dim=c["dim"], n_layers=c["layers"], n_heads=c["heads"],
                       n_kv_heads=c["kv_heads"], ffn_dim=c["ffn"])


def _gpt2_config(c):
    return GPT2Config(vocab_size=c["vocab"], dim=c["dim"], n_layers=c["layers"], n_heads=c["heads"])


def _tokens(c, vocab, gen):
    ids = torch.randint(0, vocab, (c["batch"], c["seq"] + 1), device="cuda", generator=gen)
    return ids[:, :-1].contiguous(), ids[:, 1:].contiguous()


def prepare(case, seed):
    c, kind = case, case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = _generator(seed)
    init = 1000 * (seed % 1000003)
    torch.manual_seed(init)
    if kind == "llama":
        pipe = build_llama_pipeline(_llama_config(c), c["batch"], c["seq"], c["microbatches"], dev,
                                    schedule=c["schedule"], virtual_stages=c["stages"], seed=init,
                                    activation_checkpointing=c["checkpoint"])
        ids, target = _tokens(c, c["vocab"], gen)
        return dict(kind=kind, pipe=pipe, ids=ids, target=target)
    if kind == "gpt2":
        pipe = build_gpt2_pipeline(_gpt2_config(c), c["batch"], c["seq"], c["microbatches"], dev, schedule=c["schedule"],
                                   seed=init)
        ids, target = _tokens(c, c["vocab"], gen)
        return dict(kind=kind, pipe=pipe, ids=ids, target=target)
    if kind == "score":
        model = Llama(_llama_config(c), device=dev)
        ids, target = _tokens(c, c["vocab"], gen)
        return dict(kind=kind, model=model, ids=ids, target=target)
    if kind == "attention":
        T, D = c["batch"] * c["seq"], c["head_dim"]
        qkv = torch.randn(T, (c["heads"] + 2 * c["kv_heads"]) * D, device=dev, dtype=BF16, generator=gen)
        dout = torch.randn(T, c["heads"] * D, device=dev, dtype=BF16, generator=gen)
        tables = pf.rope_tables(c["seq"], D, 10000.0, dev) if c["rotary"] else (None, None)
        return dict(kind=kind, case=c, qkv=qkv.requires_grad_(), dout=dout, tables=tables)
    if kind == "head":
        cfg = GPT2Config(vocab_size=c["vocab"], dim=c["dim"])
        rows = cfg.padded_vocab if c["family"] == "gpt2" else c["vocab"]
        h = torch.randn(c["tokens"], c["dim"], device=dev, dtype=BF16, generator=gen)
        weight = torch.nn.Parameter(0.02 * torch.randn(rows, c["dim"], device=dev, dtype=BF16, generator=gen))
        target = torch.randint(0, c["vocab"], (c["tokens"],), device=dev, generator=gen)
        target[::61] = -100  # padding tokens of a packed batch
        loss_fn = gpt2_loss(cfg) if c["family"] == "gpt2" else causal_lm_loss
        return dict(kind=kind, h=h.requires_grad_(), weight=weight, flat=FlatParams([weight]), target=target,
                    loss_fn=loss_fn)
    if kind == "moe":
        ep = EPContext(None, max_tokens=c["tokens"], hidden=c["dim"], top_k=c["top_k"], n_experts=c["experts"],
                       device=dev, capacity_factor=1.0)
        layer = MoEFeedForward(c["dim"], c["ffn"], c["experts"], c["top_k"], ep, device=dev, dtype=BF16)
        x = torch.randn(c["tokens"], c["dim"], device=dev, dtype=BF16, generator=gen)
        dy = torch.randn(c["tokens"], c["dim"], device=dev, dtype=BF16, generator=gen)
        return dict(kind=kind, layer=layer, flat=FlatParams(layer.parameters()), x=x.requires_grad_(), dy=dy)
    weight = torch.nn.Parameter(0.02 * torch.randn(c["numel"], device=dev, dtype=BF16, generator=gen))
    flat = FlatParams([weight])
    flat.grad.normal_(std=1e-2, generator=gen)
    return dict(kind=kind, flat=flat, opt=FusedAdamW(flat, lr=3e-4, weight_decay=0.1, master_weights=c["master"]))


def run(state):
    kind = state["kind"]
    if kind in ("llama", "gpt2"):
        pipe = state["pipe"]
        loss = pipe.train_step(state["ids"], state["target"])
        opt = pipe.optimizer
        return dict(loss=loss, weights=[g.data for g in opt.groups], m=opt.m, v=opt.v)
    if kind == "score":
        with torch.no_grad():
            logits = state["model"](state["ids"])
            return dict(logits=logits, loss=causal_lm_loss(logits, state["target"]))
    if kind == "attention":
        c = state["case"]
        cos, sin = state["tables"]
        qkv = state["qkv"].clone() if cos is not None else state["qkv"]  # the rotation overwrites its argument
        out = pf.rope_attention(qkv, cos, sin, c["batch"], c["seq"], c["heads"], c["kv_heads"], c["head_dim"])
        (dqkv,) = torch.autograd.grad(out, state["qkv"], state["dout"])
        return dict(out=out, dqkv=dqkv)
    if kind == "head":
        state["flat"].zero_grad()
        loss = state["loss_fn"](pf.linear(state["h"], state["weight"]), state["target"])
        (dh,) = torch.autograd.grad(loss, state["h"])
        return dict(loss=loss, dh=dh, dweight=state["flat"].grad)
    if kind == "moe":
        state["flat"].zero_grad()
        y = state["layer"](state["x"])
        (dx,) = torch.autograd.grad(y, state["x"], state["dy"])
        return dict(y=y, aux=state["layer"].last_aux_loss, dx=dx, dweights=state["flat"].grad)
    opt = state["opt"]
    opt.step(grad_scale=0.5)
    return dict(weights=opt.groups[0].data, m=opt.m[0], v=opt.v[0], master=opt.master[0])


def work(case):
    """Bytes: every input read once, every output written once.  Operations: the contractions, causal attention counted
    over the lower triangle (two products forward, five backward)."""
    c, kind = case, case["kind"]
    if kind in ("llama", "score"):
        hd = c["dim"] // c["heads"]
        layer = c["dim"] * (c["heads"] + 2 * c["kv_heads"]) * hd + c["dim"] ** 2 + 3 * c["dim"] * c["ffn"]
        head = c["vocab"] * c["dim"]
        tokens = c["batch"] * c["seq"]
        params = c["layers"] * (layer + 2 * c["dim"]) + 2 * head + c["dim"]
        if kind == "score":
            per_token = c["layers"] * (2 * layer + 2 * c["seq"] * c["dim"]) + 2 * head
            table_rows = min(tokens, c["vocab"])  # only the looked-up rows of the embedding are read
            return dict(bytes=2 * (params - head + table_rows * c["dim"]) + tokens * (2 * c["vocab"] + 16),
                        flops=tokens * per_token)
        again = 1 if c["checkpoint"] else 0
        per_token = c["layers"] * ((6 + 2 * again) * layer + (7 + 2 * again) * c["seq"] * c["dim"]) + 6 * head
        return dict(bytes=20 * params + 16 * tokens, flops=tokens * per_token)
    if kind == "gpt2":
        rows = _gpt2_config(c).padded_vocab
        tokens = c["batch"] * c["seq"]
        params = c["layers"] * (12 * c["dim"] ** 2 + 13 * c["dim"]) + (rows + 1024 + 2) * c["dim"]
        per_token = c["layers"] * (72 * c["dim"] ** 2 + 7 * c["seq"] * c["dim"]) + 6 * rows * c["dim"]
        return dict(bytes=20 * params + 16 * tokens, flops=tokens * per_token)
    if kind == "attention":
        T = c["batch"] * c["seq"]
        width_q, width_kv = c["heads"] * c["head_dim"], 2 * c["kv_heads"] * c["head_dim"]
        return dict(bytes=4 * T * (width_q + width_kv) + 4 * T * width_q, flops=7 * T * c["seq"] * width_q)
    if kind == "head":
        rows = GPT2Config(vocab_size=c["vocab"]).padded_vocab if c["family"] == "gpt2" else c["vocab"]
        return dict(bytes=6 * rows * c["dim"] + 4 * c["tokens"] * c["dim"] + 8 * c["tokens"],
                    flops=6 * c["tokens"] * c["dim"] * rows)
    if kind == "moe":
        params = 3 * c["experts"] * c["dim"] * c["ffn"]
        return dict(bytes=6 * params + 8 * c["tokens"] * c["dim"],
                    flops=18 * c["tokens"] * c["top_k"] * c["dim"] * c["ffn"])
    return dict(bytes=(30 if c["master"] else 24) * c["numel"], flops=12 * c["numel"])


def tolerance(case):
    """bf16 results against the same path in fp32 (same weights and inputs) differ by, in the 2-norm: attention 0.004, head
    0.002, whole steps and scores of two to four wide layers 0.02 (first moments; 0.025 for their squares).  Two
    implementations with other rounding points differ by that much from each other.  The expert layer is 0.004 where both
    choose the same experts.  The update alone is fp32 arithmetic; its bf16 weights may fall to the other side of a tie."""
    kind = case["kind"]
    if kind in ("llama", "gpt2", "score"):
        return {"rel": 0.03, "max": 0.99}
    if kind == "adamw":
        return {"rel": 1e-4, "max": 0.01}
    return {"rel": 0.01, "max": 0.4}


# ------------------------------------------------------------------------------------------------
# the same results in 64 bits, from plain torch operations
# ------------------------------------------------------------------------------------------------
def _again(fn, *args):
    """``fn(*args)`` without keeping its intermediates for the backward."""
    return torch.utils.checkpoint.checkpoint(fn, *args, use_reentrant=False)


def _attend64(q, k, v):  # [heads of one key group, S, D], [S, D], [S, D]
    mask = torch.ones(k.shape[0], k.shape[0], dtype=torch.bool, device=k.device).triu(1)
    return (q @ k.T / math.sqrt(k.shape[1])).masked_fill(mask, float("-inf")).softmax(-1) @ v


def _attention64(qkv, S, heads, kv_heads, hd, rotary, theta=10000.0):
    q, k, v = (t.view(-1, S, t.shape[1] // hd, hd).transpose(1, 2)
               for t in qkv.split([heads * hd, kv_heads * hd, kv_heads * hd], dim=1))
    if rotary:
        inv = theta ** (-torch.arange(0, hd, 2, dtype=torch.float64, device=qkv.device) / hd)
        ang = torch.outer(torch.arange(S, dtype=torch.float64, device=qkv.device), inv)
        c, s = ang.cos(), ang.sin()

        def rotate(x):
            a, b = x[..., : hd // 2], x[..., hd // 2:]
            return torch.cat([a * c - b * s, b * c + a * s], dim=-1)

        q, k = rotate(q), rotate(k)
    rep = heads // kv_heads
    out = [torch.cat([_again(_attend64, q[b, j * rep:(j + 1) * rep], k[b, j], v[b, j]) for j in range(kv_heads)])
           for b in range(q.shape[0])]
    return torch.stack(out).transpose(1, 2).reshape(-1, heads * hd)


def _llama64(c, w, ids):
    """Logits of one batch; ``w`` holds the weights by name."""
    hd = c["dim"] // c["heads"]

    def norm(x, g):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * g

    def layer(x, i):
        n = f"layers.{i}."
        qkv = norm(x, w[n + "attention_norm.weight"]) @ w[n + "attention.wqkv.weight"].T
        x = x + _attention64(qkv, ids.shape[1], c["heads"], c["kv_heads"], hd, True) @ w[n + "attention.wo.weight"].T
        g, u = (norm(x, w[n + "ffn_norm.weight"]) @ w[n + "feed_forward.w_gate_up.weight"].T).chunk(2, dim=-1)
        return x + (torch.nn.functional.silu(g) * u) @ w[n + "feed_forward.w_down.weight"].T

    x = w["tok_embeddings.weight"][ids.reshape(-1)]
    for i in range(c["layers"]):
        x = _again(layer, x, i)
    return norm(x, w["norm.weight"]) @ w["output.weight"].T


def _gpt264(c, w, ids):
    def norm(x, n):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w[n + ".weight"], w[n + ".bias"], 1e-5)

    def lin(x, n):
        return x @ w[n + ".weight"].T + w[n + ".bias"]

    def layer(x, i):
        n = f"h.{i}."
        qkv = lin(norm(x, n + "ln_1"), n + "attn_c_attn")
        x = x + lin(_attention64(qkv, ids.shape[1], c["heads"], c["heads"], 64, False), n + "attn_c_proj")
        h = torch.nn.functional.gelu(lin(norm(x, n + "ln_2"), n + "mlp_c_fc"), approximate="tanh")
        return x + lin(h, n + "mlp_c_proj")

    x = w["wte.weight"][ids.reshape(-1)] + w["wte.positions"][: ids.shape[1]].repeat(ids.shape[0], 1)
    for i in range(c["layers"]):
        x = _again(layer, x, i)
    return (norm(x, "ln_f") @ w["wte.weight"].T)[:, : c["vocab"]]


def _adamw64(w, grad, lr, betas, eps, decay):
    """(weights, m, v) after the first step."""
    m, v = (1 - betas[0]) * grad, (1 - betas[1]) * grad ** 2
    return w * (1 - lr * decay) - lr * grad / (grad.abs() + eps), m, v


def _step64(c, state):
    pipe = state["pipe"]
    opt = pipe.optimizer
    params = {n: p for s in pipe.stages for n, p in s.submod.named_parameters()}
    w = {n: p.detach().double().requires_grad_() for n, p in params.items()}
    loss = 0.0
    for b in range(c["batch"]):  # every sequence has the same number of targets: the mean of means is the mean
        logits = (_llama64 if c["kind"] == "llama" else _gpt264)(c, w, state["ids"][b:b + 1])
        part = torch.nn.functional.cross_entropy(logits, state["target"][b]) / c["batch"]
        part.backward()
        loss = loss + part.detach()
    names = {id(p): n for n, p in params.items()}
    weights, ms, vs = [], [], []
    for g in opt.groups:
        flat = g.data.double()
        grad = torch.zeros_like(flat)
        for p, o in zip(g.params, g.offsets):
            grad[o:o + p.numel()] = w[names[id(p)]].grad.reshape(-1)
        new = _adamw64(flat, grad, opt.lr, opt.betas, opt.eps, opt.weight_decay)
        for out, x in zip((weights, ms, vs), new):
            out.append(x)
    return dict(loss=loss, weights=weights, m=ms, v=vs)


def _moe64(c, state):
    layer, x, dy = state["layer"], state["x"].detach().double(), state["dy"].double()
    E, k, f = c["experts"], c["top_k"], c["ffn"]
    router = layer.router.detach().double()
    x.requires_grad_()
    router.requires_grad_()
    logits = (x @ router.T)[:, :E]
    probs = logits.softmax(-1)
    # the choice is made on logits of the layer's own 16 bits: a near tie is not a matter of precision
    chosen = torch.sort(logits.detach().to(BF16).float(), dim=-1, descending=True, stable=True).indices[:, :k]
    topw = probs.gather(1, chosen)
    topw = topw / topw.sum(-1, keepdim=True)
    share = torch.bincount(chosen.reshape(-1), minlength=E).double() / chosen.numel()
    aux = E * (share * probs.mean(0)).sum()
    y = torch.zeros_like(x)
    dx = torch.zeros_like(x)
    dtopw = torch.zeros_like(topw)
    dgu, dd = [], []
    for e in range(E):
        tok, slot = (chosen == e).nonzero(as_tuple=True)
        xe = x.detach()[tok].requires_grad_()
        gu = layer.w_gate_up[e].detach().double().requires_grad_()
        down = layer.w_down[e].detach().double().requires_grad_()
        we = topw.detach()[tok, slot].requires_grad_()
        g, u = (xe @ gu.T).split(f, dim=1)
        ye = (torch.nn.functional.silu(g) * u) @ down.T * we[:, None]
        gx, gw, ggu, gd = torch.autograd.grad(ye, [xe, we, gu, down], dy[tok])
        y = y.index_add(0, tok, ye.detach())
        dx = dx.index_add(0, tok, gx)
        dtopw[tok, slot] = gw
        dgu.append(ggu.float())  # 2.8 GB an expert in 64 bits
        dd.append(gd.float())
    rx, drouter = torch.autograd.grad([topw, aux], [x, router], [dtopw, torch.full_like(aux, layer.aux_coef)])
    grads = [drouter.float().reshape(-1)] + [g.reshape(-1) for g in dgu] + [g.reshape(-1) for g in dd]
    return dict(y=y, aux=aux.detach(), dx=dx + rx, dweights=torch.cat(grads))


def exact(case, seed):
    c, kind, state = case, case["kind"], prepare(case, seed)
    if kind in ("llama", "gpt2"):
        return _step64(c, state)
    if kind == "score":
        with torch.no_grad():
            w = {n: p.double() for n, p in state["model"].named_parameters()}
            logits = _llama64(c, w, state["ids"])
            loss = torch.nn.functional.cross_entropy(logits, state["target"].reshape(-1))
            return dict(logits=logits.view(c["batch"], c["seq"], -1), loss=loss)
    if kind == "attention":
        qkv = state["qkv"].detach().double().requires_grad_()
        out = _attention64(qkv, c["seq"], c["heads"], c["kv_heads"], c["head_dim"], c["rotary"])
        (dqkv,) = torch.autograd.grad(out, qkv, state["dout"].double())
        return dict(out=out.detach(), dqkv=dqkv)
    if kind == "head":
        h = state["h"].detach().double().requires_grad_()
        weight = state["weight"].detach().double().requires_grad_()
        loss = torch.nn.functional.cross_entropy((h @ weight.T)[:, : c["vocab"]], state["target"])
        dh, dw = torch.autograd.grad(loss, [h, weight])
        return dict(loss=loss.detach(), dh=dh, dweight=dw.reshape(-1))
    if kind == "moe":
        return _moe64(c, state)
    opt = state["opt"]
    flat = opt.groups[0]
    master = opt.master[0]
    w = flat.data.double() if master is None else master.double()
    w, m, v = _adamw64(w, flat.grad.double() * 0.5, opt.lr, opt.betas, opt.eps, opt.weight_decay)
    return dict(weights=w, m=m, v=v, master=None if master is None else w)
