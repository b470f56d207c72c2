"""The workloads whose speed this repository follows, as plain data plus one function each to
make their inputs, run them once through the public entry points, and state what they need.

The sizes come from the repository's own configurations: the Llama-7B layer (hidden 4096,
FFN 11008, 32 heads of 128, vocabulary 32000, sequences up to 2048), GPT-2 medium (width 1024,
16 heads of 64, vocabulary 50257, sequence 1024, micro-batch 8), gradient buckets of the
low-bit collectives (4 and 8 bit, block 256) and the tiny test models.  ``listed()`` names the
points that are followed by name; ``draw(rng)`` gives more points of the same ranges.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from bitscom_b200 import quantization as Q
from bitscom_b200.models.gpt2 import GPT2, GPT2Config
from bitscom_b200.models.llama import LlamaConfig, LlamaStage
from bitscom_b200.ops import attention as A
from bitscom_b200.ops import gemm as G
from bitscom_b200.ops import nn as K
from bitscom_b200.parallel import fused

BLOCK = 256          # quantization block of every low-bit path's default
QMAX = {4: 7, 8: 127}
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
SIZE = {"fp32": 4, "bf16": 2}


def listed():
    return [
        # one small parameter's gradient through the codec: latency and launches
        dict(name="codec_small", op="codec", numel=4097, bits=4, dtype="fp32", stochastic=False),
        # a 25 MB-class data-parallel bucket in bf16 at 8 bit, with a ragged tail
        dict(name="codec_bucket_bf16", op="codec", numel=6553611, bits=8, dtype="bf16",
             stochastic=False),
        # a 256 MB fp32 bucket at 4 bit with stochastic rounding, the trainers' setting
        dict(name="codec_large_sr", op="codec", numel=1 << 26, bits=4, dtype="fp32",
             stochastic=True),
        # the fused all-reduce kernel: what four workers' buckets of 32 Mi elements cost
        dict(name="allreduce_4_workers", op="allreduce", world=4, numel=32 << 20, bits=4,
             dtype="bf16", stochastic=True),
        # causal attention of the Llama layer, training direction (two sequences of 2048)
        dict(name="attention_llama", op="attention", batch=2, seq=2048, heads=32, head_dim=128,
             backward=True),
        # causal attention of GPT-2 medium, micro-batch 8, training direction
        dict(name="attention_gpt2", op="attention", batch=8, seq=1024, heads=16, head_dim=64,
             backward=True),
        # scoring one short sequence: forward only, too few query blocks to fill the chip
        dict(name="attention_short_fwd", op="attention", batch=1, seq=384, heads=12, head_dim=64,
             backward=False),
        # one projection of a short ragged batch (fine-tuning of single documents), both ways
        dict(name="linear_ragged", op="linear", tokens=200, inner=1024, outer=3072),
        # final norm + LM head + loss over a 32000-word vocabulary, both ways
        dict(name="llama_head", op="head", tokens=4096, hidden=4096, vocab=32000),
        # scoring a 128-token prompt: two full-width layers and the head, logits out
        dict(name="llama_prompt", op="prompt", batch=1, seq=128, layers=2),
        # one micro-batch of GPT-2 medium at reduced depth: loss and every gradient
        dict(name="gpt2_step", op="gpt2", batch=8, seq=1024, layers=2),
        # one decoder layer of the 7B model, forward and backward, a micro-batch of two
        dict(name="llama_layer", op="layer", batch=2, seq=2048),
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["codec", "codec", "allreduce", "attention", "attention", "linear", "linear",
                     "head", "prompt", "gpt2", "layer"])
    if op == "codec":
        return dict(op=op, numel=_log_between(rng, 4096, 1 << 26) | rng.choice([0, 1]),
                    bits=rng.choice([4, 8]), dtype=rng.choice(["fp32", "bf16"]),
                    stochastic=rng.choice([False, True]))
    if op == "allreduce":
        return dict(op=op, world=rng.choice([2, 4, 8]), numel=_log_between(rng, 1 << 18, 16 << 20),
                    bits=rng.choice([4, 8]), dtype=rng.choice(["fp32", "bf16"]),
                    stochastic=rng.choice([False, True]))
    if op == "attention":
        head_dim = rng.choice([64, 128])
        seq = 128 * _log_between(rng, 1, 16)
        batch = rng.randint(1, max(1, 8192 // seq) if seq > 512 else 8)
        heads = rng.randint(1, 32 if batch * seq <= 4096 else 16)
        return dict(op=op, batch=batch, seq=seq, heads=heads, head_dim=head_dim,
                    backward=rng.choice([False, True, True]))
    if op == "linear":
        inner, outer = rng.choice([(1024, 3072), (1024, 1024), (1024, 4096), (4096, 1024),
                                   (4096, 4096), (256, 768), (11008, 4096)])
        return dict(op=op, tokens=_log_between(rng, 64, 8192), inner=inner, outer=outer)
    if op == "head":
        hidden, vocab = rng.choice([(4096, 32000), (1024, 50432), (256, 512)])
        return dict(op=op, tokens=_log_between(rng, 100, 4096), hidden=hidden, vocab=vocab)
    if op == "prompt":
        return dict(op=op, batch=rng.randint(1, 4), seq=128 * rng.randint(1, 4),
                    layers=rng.randint(1, 2))
    if op == "gpt2":
        return dict(op=op, batch=rng.randint(1, 8), seq=128 * rng.randint(1, 8),
                    layers=rng.randint(1, 2))
    return dict(op=op, batch=rng.randint(1, 2), seq=128 * rng.randint(1, 16))


# ----------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(dtype)


def _codec_input(case, seed):
    # gradients: small, and of another magnitude from block to block
    gen = _generator(seed)
    n = case["numel"]
    x = torch.randn(n, device="cuda", generator=gen)
    blocks = -(-n // BLOCK)
    spread = torch.exp(torch.randn(blocks, device="cuda", generator=gen))
    x *= 1e-3 * spread.repeat_interleave(BLOCK)[:n]
    return x.to(DTYPES[case["dtype"]])


def _allreduce_inputs(case, seed):
    gen = _generator(seed)
    return [_randn(gen, case["numel"], std=1e-3, dtype=DTYPES[case["dtype"]])
            for _ in range(case["world"])]


def _attention_inputs(case, seed):
    gen = _generator(seed)
    tokens, width = case["batch"] * case["seq"], case["heads"] * case["head_dim"]
    qkv = _randn(gen, tokens, 3 * width)
    d_out = _randn(gen, tokens, width, std=1e-2) if case["backward"] else None
    return qkv, d_out


def _linear_inputs(case, seed):
    gen = _generator(seed)
    return (_randn(gen, case["tokens"], case["inner"]),
            _randn(gen, case["outer"], case["inner"], std=0.02),
            _randn(gen, case["tokens"], case["outer"], std=1e-2))


def _head_inputs(case, seed):
    gen = _generator(seed)
    T, H, V = case["tokens"], case["hidden"], case["vocab"]
    x = _randn(gen, T, H)
    norm = (1 + 0.1 * torch.randn(H, device="cuda", generator=gen)).to(torch.bfloat16)
    head = _randn(gen, V, H, std=0.02)
    targets = torch.randint(1, V, (T,), device="cuda", generator=gen)
    targets[::17] = 0  # padding, ignored by the loss
    return x, norm, head, targets


def _prompt_config(case):
    return LlamaConfig(num_layers=case["layers"])


def _gpt2_config(case):
    return GPT2Config(n_layer=case["layers"], seq=case["seq"])


def _token_ids(case, seed, vocab):
    gen = _generator(int(seed) + 1)
    return torch.randint(1, vocab, (case["batch"], case["seq"]), device="cuda", generator=gen)


def _layer_inputs(case, seed, hidden):
    gen = _generator(int(seed) + 1)
    tokens = case["batch"] * case["seq"]
    return _randn(gen, tokens, hidden), _randn(gen, tokens, hidden, std=1e-2)


def _layer_stage(seed):
    # a middle stage of a pipeline split owns exactly one decoder layer
    return LlamaStage(LlamaConfig(num_layers=3), stage=1, num_stages=3, seed=seed)


def prepare(case, seed):
    op = case["op"]
    state = {"case": case}
    if op == "codec":
        state["x"] = _codec_input(case, seed)
    elif op == "allreduce":
        state["grads"] = _allreduce_inputs(case, seed)
        state["group"] = fused.EmulatedWorld(case["world"], "cuda:0", region_bytes=64 << 20)
    elif op == "attention":
        qkv, state["d_out"] = _attention_inputs(case, seed)
        state["qkv"] = qkv.requires_grad_(case["backward"])
    elif op == "linear":
        x, w, state["dy"] = _linear_inputs(case, seed)
        state["x"] = x.requires_grad_()
        state["w"] = torch.nn.Parameter(w)
        state["w"].main_grad = torch.zeros(w.shape, dtype=torch.float32, device="cuda")
    elif op == "head":
        x, norm, head, state["targets"] = _head_inputs(case, seed)
        state["x"] = x.requires_grad_()
        for name, value in (("norm", norm), ("head", head)):
            state[name] = torch.nn.Parameter(value)
            state[name].main_grad = torch.zeros(value.shape, dtype=torch.float32, device="cuda")
    elif op == "prompt":
        cfg = _prompt_config(case)
        state["model"] = LlamaStage(cfg, seed=seed)
        state["ids"] = _token_ids(case, seed, cfg.vocab_size)
    elif op == "gpt2":
        cfg = _gpt2_config(case)
        state["model"] = GPT2(cfg, seed=seed)
        state["ids"] = _token_ids(case, seed, cfg.vocab_size)
    else:
        state["model"] = _layer_stage(seed)
        x, state["dy"] = _layer_inputs(case, seed, state["model"].cfg.hidden_size)
        state["x"] = x.requires_grad_()
    return state


# ----------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    op = case["op"]
    if op == "codec":
        x = state["x"]
        packed, scales, n = Q.quantize_pack_tensor_blockwise(
            x, case["bits"], block_size=BLOCK, stochastic_rounding=case["stochastic"],
            sr_seed=7)
        y = Q.unpack_dequantize_tensor_blockwise(packed, scales, case["bits"], n,
                                                 block_size=BLOCK, dtype=x.dtype)
        return packed, scales, y
    if op == "allreduce":
        # the all-reduce works in place; the workers' own gradients are kept
        out = [g.clone() for g in state["grads"]]
        state["group"].all_reduce(out, bitwidth=case["bits"], block_size=BLOCK,
                                  stochastic=case["stochastic"], seed=7)
        return out
    if op == "attention":
        args = (case["batch"], case["seq"], case["heads"], case["head_dim"])
        if not case["backward"]:
            with torch.no_grad():
                return A.attention(state["qkv"], *args)
        out = A.attention(state["qkv"], *args)
        (dqkv,) = torch.autograd.grad(out, state["qkv"], state["d_out"])
        return out, dqkv
    if op == "linear":
        x, w = state["x"], state["w"]
        w.main_grad.zero_()
        x.grad = None
        y = G.linear(x, w)
        y.backward(state["dy"])
        return y.detach(), x.grad, w.main_grad
    if op == "head":
        x, norm, head = state["x"], state["norm"], state["head"]
        norm.main_grad.zero_()
        head.main_grad.zero_()
        x.grad = None
        h = K.rmsnorm(x, norm)
        loss = K.cross_entropy(G.linear(h, head), state["targets"], ignore_index=0)
        loss.backward()
        return loss.detach(), x.grad, norm.main_grad, head.main_grad
    if op == "prompt":
        with torch.no_grad():
            return state["model"](state["ids"])
    if op == "gpt2":
        model = state["model"]
        model.flat.grads.zero_()
        loss = model(state["ids"], state["ids"])
        loss.backward()
        model.collect_autograd_grads()
        return loss.detach(), model.flat.grads
    model, x = state["model"], state["x"]
    model.flat.grads.zero_()
    x.grad = None
    y = model.layer(1, x, case["batch"], case["seq"])
    y.backward(state["dy"])
    return y.detach(), x.grad, model.flat.grads


# ----------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------

def _llama_layer_params(cfg):
    return 4 * cfg.hidden_size ** 2 + 3 * cfg.hidden_size * cfg.intermediate_size


def _attention_flops(batch, seq, heads, head_dim, backward):
    # causal: half of the score matrix; forward has two products of it, backward five
    one = 2 * batch * heads * head_dim * seq * (seq + 1) // 2
    return one * (2 + (5 if backward else 0))


def work(case):
    op = case["op"]
    if op == "codec":
        n = case["numel"]
        wire = n * case["bits"] / 8 + 2 * (-(-n // BLOCK))
        return {"bytes": 2 * n * SIZE[case["dtype"]] + 2 * wire, "flops": 10 * n}
    if op == "allreduce":
        W, n = case["world"], case["numel"]
        wire = n * (case["bits"] / 8 + 2 / BLOCK)
        # every worker: its gradients read, its packed shards written and read, the reduced
        # shards written to and read by all, the result written
        return {"bytes": W * (2 * n * SIZE[case["dtype"]] + 4 * wire), "flops": 30 * n * W}
    if op == "attention":
        T, H = case["batch"] * case["seq"], case["heads"] * case["head_dim"]
        nbytes = 2 * T * 4 * H
        if case["backward"]:
            nbytes += 2 * T * 4 * H
        return {"bytes": nbytes, "flops": _attention_flops(
            case["batch"], case["seq"], case["heads"], case["head_dim"], case["backward"])}
    if op == "linear":
        T, I, O = case["tokens"], case["inner"], case["outer"]
        return {"bytes": 2 * (2 * T * I + 2 * T * O + O * I) + 4 * O * I, "flops": 6 * T * I * O}
    if op == "head":
        T, H, V = case["tokens"], case["hidden"], case["vocab"]
        return {"bytes": 2 * (2 * T * H + V * H) + 4 * V * H, "flops": 6 * T * H * V}
    if op == "prompt":
        cfg = _prompt_config(case)
        T = case["batch"] * case["seq"]
        params = cfg.num_layers * _llama_layer_params(cfg) + cfg.vocab_size * cfg.hidden_size
        return {"bytes": 2 * (params + T * cfg.vocab_size),
                "flops": 2 * T * params + cfg.num_layers * _attention_flops(
                    case["batch"], case["seq"], cfg.num_heads, cfg.head_dim, False)}
    if op == "gpt2":
        cfg = _gpt2_config(case)
        T = case["batch"] * case["seq"]
        layer = 12 * cfg.d_model ** 2
        params = cfg.n_layer * layer + cfg.padded_vocab * cfg.d_model
        return {"bytes": 6 * params, "flops": 6 * T * params + cfg.n_layer * _attention_flops(
            case["batch"], case["seq"], cfg.n_head, cfg.d_model // cfg.n_head, True)}
    cfg = LlamaConfig()
    T = case["batch"] * case["seq"]
    params = _llama_layer_params(cfg)
    return {"bytes": 6 * params + 2 * T * 4 * cfg.hidden_size,
            "flops": 6 * T * params + _attention_flops(case["batch"], case["seq"], cfg.num_heads,
                                                       cfg.head_dim, True)}


def tolerance(case):
    op = case["op"]
    if op in ("codec", "allreduce"):
        return "exact"   # codes, scales and the order of the sums are part of the wire contract
    # bf16 results of fp32 accumulations: about four times the distance to 64 bits (measured:
    # attention 0.0024, one projection 0.0017, head 0.0023, a layer 0.0065, GPT-2's gradients
    # 0.0073, two whole layers plus head 0.013 because their logits are small differences)
    return {"rel": {"attention": 1e-2, "linear": 7e-3, "head": 1e-2, "layer": 2.5e-2,
                    "gpt2": 3e-2, "prompt": 5e-2}[op]}


# ----------------------------------------------------------------------------------
# the same results in 64 bits
# ----------------------------------------------------------------------------------

def _exact_codec(case, seed):
    if case["stochastic"]:
        return None  # the codes depend on the random stream
    x = _codec_input(case, seed).double()
    n, blocks = x.numel(), -(-x.numel() // BLOCK)
    padded = F.pad(x, (0, blocks * BLOCK - n)).view(blocks, BLOCK)
    scales = padded.abs().amax(1) / QMAX[case["bits"]]
    # the stored scale is fp16: the values are multiples of the rounded one
    s16 = torch.where(scales > 0, scales, torch.ones_like(scales)).half().double()
    codes = torch.round(padded / s16[:, None]).clamp(-QMAX[case["bits"]] - 1, QMAX[case["bits"]])
    codes = torch.where(codes.isfinite(), codes, torch.zeros_like(codes))
    return None, scales, (codes * s16[:, None]).view(-1)[:n]


def _exact_attention_head(q, k, v, d_out):
    scale = 1.0 / math.sqrt(q.shape[-1])
    seq = q.shape[0]
    keep = torch.ones(seq, seq, dtype=torch.bool, device=q.device).tril()
    p = torch.softmax((q @ k.t() * scale).masked_fill(~keep, float("-inf")), -1)
    o = p @ v
    if d_out is None:
        return o, None, None, None
    dv = p.t() @ d_out
    ds = p * (d_out @ v.t() - (d_out * o).sum(-1, keepdim=True)) * scale
    return o, ds @ k, ds.t() @ q, dv


def _exact_attention(case, qkv, d_out):
    B, S, nh, hd = case["batch"], case["seq"], case["heads"], case["head_dim"]
    q5 = qkv.double().view(B, S, 3, nh, hd)
    out = torch.empty(B, S, nh, hd, dtype=torch.float64, device=qkv.device)
    grad = torch.empty_like(q5) if d_out is not None else None
    g4 = d_out.double().view(B, S, nh, hd) if d_out is not None else None
    for b in range(B):
        for h in range(nh):
            o, dq, dk, dv = _exact_attention_head(
                q5[b, :, 0, h], q5[b, :, 1, h], q5[b, :, 2, h],
                None if g4 is None else g4[b, :, h])
            out[b, :, h] = o
            if grad is not None:
                grad[b, :, 0, h], grad[b, :, 1, h], grad[b, :, 2, h] = dq, dk, dv
    out = out.view(B * S, nh * hd)
    return out if grad is None else (out, grad.view(B * S, 3 * nh * hd))


class _Attention64(torch.autograd.Function):
    """Causal attention over [tokens, 3 * width], one head at a time (memory)."""

    @staticmethod
    def forward(ctx, qkv, case):
        ctx.case = case
        ctx.save_for_backward(qkv)
        return _exact_attention(case, qkv, None)

    @staticmethod
    def backward(ctx, d_out):
        (qkv,) = ctx.saved_tensors
        return _exact_attention(ctx.case, qkv, d_out)[1], None


def _rms64(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _exact_head(case, seed):
    x, norm, head, targets = _head_inputs(case, seed)
    x, norm, head = (t.double().requires_grad_() for t in (x, norm, head))
    loss = F.cross_entropy(_rms64(x, norm) @ head.t(), targets, ignore_index=0)
    loss.backward()
    return loss.detach(), x.grad, norm.grad, head.grad


def _rope64(t, seq, heads, head_dim, theta):
    half = head_dim // 2
    inv = 1.0 / theta ** (torch.arange(0, head_dim, 2, dtype=torch.float64, device=t.device)
                          / head_dim)
    ang = torch.outer(torch.arange(seq, dtype=torch.float64, device=t.device), inv)
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]
    t = t.view(-1, seq, heads, head_dim)
    a, b = t[..., :half], t[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1).reshape(-1, heads * head_dim)


def _llama_layer64(cfg, w, x, batch, seq):
    H, nh, hd = cfg.hidden_size, cfg.num_heads, cfg.head_dim
    qkv = _rms64(x, w["norm1"], cfg.rms_eps) @ w["wqkv"].t()
    q, k, v = qkv[:, :H], qkv[:, H:2 * H], qkv[:, 2 * H:]
    qkv = torch.cat([_rope64(q, seq, nh, hd, cfg.rope_theta),
                     _rope64(k, seq, nh, hd, cfg.rope_theta), v], 1)
    shape = dict(batch=batch, seq=seq, heads=nh, head_dim=hd)
    x = x + _Attention64.apply(qkv, shape) @ w["wo"].t()
    gate, up = (_rms64(x, w["norm2"], cfg.rms_eps) @ w["wgu"].t()).chunk(2, 1)
    return x + (F.silu(gate) * up) @ w["wdown"].t()


def _flat_weights64(flat, needs_grad):
    return {name: view.detach().double().requires_grad_(needs_grad)
            for name, view in flat.named_views()}


def _flat_grads64(flat, weights):
    out = torch.zeros(flat.numel, dtype=torch.float64, device="cuda")
    for name, (off, n, _) in flat.offsets.items():
        out[off:off + n] = weights[name].grad.reshape(-1)
    return out


def _exact_layer(case, seed):
    stage = _layer_stage(seed)
    x, dy = _layer_inputs(case, seed, stage.cfg.hidden_size)
    x = x.double().requires_grad_()
    w = _flat_weights64(stage.flat, True)
    layer = {name[len("l1."):]: t for name, t in w.items()}
    y = _llama_layer64(stage.cfg, layer, x, case["batch"], case["seq"])
    y.backward(dy.double())
    return y.detach(), x.grad, _flat_grads64(stage.flat, w)


def _exact_prompt(case, seed):
    cfg = _prompt_config(case)
    w = _flat_weights64(LlamaStage(cfg, seed=seed).flat, False)
    x = w["embed"][_token_ids(case, seed, cfg.vocab_size).reshape(-1)]
    for i in range(cfg.num_layers):
        layer = {name[len(f"l{i}."):]: t for name, t in w.items() if name.startswith(f"l{i}.")}
        x = _llama_layer64(cfg, layer, x, case["batch"], case["seq"])
    logits = _rms64(x, w["final_norm"], cfg.rms_eps) @ w["embed"].t()
    return logits.view(case["batch"], case["seq"], -1)


def _exact_gpt2(case, seed):
    cfg = _gpt2_config(case)
    flat = GPT2(cfg, seed=seed).flat
    w = _flat_weights64(flat, True)
    ids = _token_ids(case, seed, cfg.vocab_size)
    B, S = ids.shape
    D, nh = cfg.d_model, cfg.n_head
    shape = dict(batch=B, seq=S, heads=nh, head_dim=D // nh)
    x = w["wte"][ids.reshape(-1)] + w["wpe"][:S].repeat(B, 1)
    for i in range(cfg.n_layer):
        p = {name[len(f"h{i}."):]: t for name, t in w.items() if name.startswith(f"h{i}.")}
        h = F.layer_norm(x, (D,), p["ln1_w"], p["ln1_b"])
        a = _Attention64.apply(h @ p["wqkv"].t() + p["bqkv"], shape)
        x = x + a @ p["wo"].t() + p["bo"]
        h = F.layer_norm(x, (D,), p["ln2_w"], p["ln2_b"])
        h = F.gelu(h @ p["wfc"].t() + p["bfc"], approximate="tanh")
        x = x + h @ p["wproj"].t() + p["bproj"]
    logits = F.layer_norm(x, (D,), w["lnf_w"], w["lnf_b"]) @ w["wte"].t()
    shifted = torch.full_like(ids, -100)
    shifted[:, :-1] = ids[:, 1:]
    loss = F.cross_entropy(logits, shifted.reshape(-1))
    loss.backward()
    return loss.detach(), _flat_grads64(flat, w)


def exact(case, seed):
    op = case["op"]
    if op == "codec":
        return _exact_codec(case, seed)
    if op == "allreduce":
        return None  # two quantizations with their own random streams lie in between
    if op == "attention":
        return _exact_attention(case, *_attention_inputs(case, seed))
    if op == "linear":
        x, w, dy = (t.double() for t in _linear_inputs(case, seed))
        return x @ w.t(), dy @ w, dy.t() @ x
    if op == "head":
        return _exact_head(case, seed)
    if op == "prompt":
        return _exact_prompt(case, seed)
    if op == "gpt2":
        return _exact_gpt2(case, seed)
    return _exact_layer(case, seed)
