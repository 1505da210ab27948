"""The work that users of this framework have it do on one GPU, as cases that can be timed and compared.

Four kinds of case, each through the public entry points:

``train``      one optimisation step of a GPT-2 or LLaMA-3 model as the trainers and the benchmark take it: zero the
               gradients, bf16-autocast forward, cross-entropy, backward, AdamW; eager or as a captured whole step,
               with the residual stream in bf16 or fp32, all weights or LoRA adapters only
``eval``       logits of a batch without gradients: validation, and the text sampler, which runs the whole window
               again for every token
``attention``  causal self-attention on a packed QKV projection, forward and backward, with and without RoPE and
               grouped-query heads: what long contexts are made of
``head``       output projection and cross-entropy over a real vocabulary, forward and backward

Depth is cut where a full model would only repeat the same layer; widths, heads, feed-forward sizes and vocabularies
are those of the model configurations (smaller vocabularies where the head has a case of its own).
"""
from __future__ import annotations

import torch
import torch.utils.checkpoint

from infinitrain_b200.autocast import AutocastGuard
from infinitrain_b200.datatype import DataType
from infinitrain_b200.device import DeviceType
from infinitrain_b200.models import GPT2, LLaMA3, gpt2_config, llama3_config
from infinitrain_b200.nn import CrossEntropyLoss, init, lora
from infinitrain_b200.ops import functional as ops
from infinitrain_b200.optim import Adam
from infinitrain_b200.parallel import global_env as genv
from infinitrain_b200.parallel.process_group import ProcessGroupFactory
from infinitrain_b200.utils.cuda_graph import GraphedTrainStep

LORA_RANK = 16


def _train(name, model, layers, batch, seq, vocab=50257, residual="bf16", graph=False, lora_rank=0):
    return {"name": name, "kind": "train", "model": model, "layers": layers, "vocab": vocab, "batch": batch, "seq": seq,
            "residual": residual, "graph": graph, "lora_rank": lora_rank}


def _eval(name, model, layers, batch, seq, vocab=50257):
    return {"name": name, "kind": "eval", "model": model, "layers": layers, "vocab": vocab, "batch": batch, "seq": seq}


def _attention(name, batch, seq, heads, kv_heads, head_dim, rope):
    return {"name": name, "kind": "attention", "batch": batch, "seq": seq, "heads": heads, "kv_heads": kv_heads,
            "head_dim": head_dim, "rope": rope}


def _head(name, tokens, width, vocab):
    return {"name": name, "kind": "head", "tokens": tokens, "width": width, "vocab": vocab}


def listed():
    return [
        # the smallest training batch of the configurations: 4 x 64 tokens of GPT-2 124M, launched op by op
        _train("gpt2 train 4x64", "gpt2", 12, 4, 64),
        # the benchmark's step: GPT-2 124M, 16 x 1024 tokens, captured as one CUDA graph
        _train("gpt2 train 16x1024 graph", "gpt2", 12, 16, 1024, graph=True),
        # documents that are not cut to a power of two, the reference's fp32 residual stream, op by op
        _train("gpt2 train 3x777 fp32 stream", "gpt2", 12, 3, 777, residual="fp32"),
        # LLaMA-3 1B layers at the context that its configuration trains with
        _train("llama-1b train 1x2048", "llama3-1b", 4, 1, 2048, vocab=32768),
        # LoRA fine-tune of LLaMA-3 8B layers: rank 16 on the attention projections, frozen base
        _train("llama-8b lora 2x2048", "llama3-8b", 2, 2, 2048, vocab=8192, lora_rank=LORA_RANK),
        # the text sampler: one short window, where latency and launches are everything
        _eval("gpt2 sample 1x96", "gpt2", 12, 1, 96),
        # validation batch of the next larger GPT-2
        _eval("gpt2-medium eval 8x1024", "gpt2-medium", 12, 8, 1024),
        # validation on sequences of an odd length
        _eval("llama-1b eval 2x1001", "llama3-1b", 4, 2, 1001, vocab=32768),
        # attention of one GPT-2 124M layer in the benchmark's batch
        _attention("attention 16x1024 12h d64", 16, 1024, 12, 12, 64, False),
        # attention of one LLaMA-3 8B layer over its whole context window
        _attention("attention 1x8192 32/8h d128", 1, 8192, 32, 8, 128, True),
        # attention of a LLaMA-3 3B layer over a few short, ragged sequences
        _attention("attention 3x200 24/8h d128", 3, 200, 24, 8, 128, True),
        # output projection and loss of LLaMA-3 1B: the 128256-wide vocabulary
        _head("head 2048x2048x128256", 2048, 2048, 128256),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["train", "train", "eval", "attention", "attention", "head"])
        if kind in ("train", "eval"):
            model = rng.choice(["gpt2", "gpt2", "gpt2-medium", "llama3-1b", "llama3-3b"])
            gpt = model.startswith("gpt2")
            seq = _log_uniform(rng, 32, 1024 if gpt else 2048)
            batch = _log_uniform(rng, 1, 16)
            layers = rng.randint(2, 12) if gpt else rng.randint(1, 3)
            vocab = 50257 if gpt else rng.choice([8192, 32000, 32768])
            if kind == "eval":
                case = _eval("", model, layers, batch, seq, vocab)
            else:
                case = _train("", model, layers, batch, seq, vocab, residual=rng.choice(["bf16", "bf16", "fp32"]),
                              graph=rng.random() < 0.4, lora_rank=0 if gpt else rng.choice([0, 0, 8, LORA_RANK]))
        elif kind == "attention":
            head_dim = rng.choice([64, 128])
            kv_heads, group = rng.choice([(12, 1), (16, 1), (20, 1), (25, 1), (8, 4), (8, 3), (1, 4)])
            case = _attention("", _log_uniform(rng, 1, 16), _log_uniform(rng, 64, 8192), kv_heads * group, kv_heads,
                              head_dim, group > 1)
        else:
            width, vocab = rng.choice([(768, 50257), (1024, 50257), (1600, 50257), (2048, 128256), (3072, 128256)])
            case = _head("", _log_uniform(rng, 64, 8192), width, vocab)
        if work(case)["flops"] <= most and work(case)["bytes"] < 12e9:
            del case["name"]
            return case


# --------------------------------------------------------------------------- building what a program keeps
def _config(case):
    make = gpt2_config if case["model"].startswith("gpt2") else llama3_config
    over = {"n_layer": case["layers"], "vocab_size": case["vocab"], "original_vocab_size": case["vocab"]}
    return make(case["model"], **over)


def _environment():
    """One rank on one GPU."""
    if genv.GlobalEnv.Instance().initialized:
        return
    genv.InitAllEnv(world_size=1, rank=0)
    ProcessGroupFactory.Instance().Init()


def _build_model(case, seed, device):
    init.manual_seed(seed)
    cls = GPT2 if case["model"].startswith("gpt2") else LLaMA3
    residual = torch.float32 if case.get("residual") == "fp32" else torch.bfloat16
    with torch.device(device):
        model = cls(case["model"], n_layer=case["layers"], vocab_size=case["vocab"], original_vocab_size=case["vocab"],
                    residual_dtype=residual)
    return model.to(device)


def prepare(case, seed):
    _environment()
    device = torch.device("cuda", 0)
    gen = torch.Generator(device=device).manual_seed(seed)
    state = {"case": case}
    if case["kind"] in ("train", "eval"):
        shape = (case["batch"], case["seq"])
        state["x"] = torch.randint(0, case["vocab"], shape, device=device, generator=gen)
        state["y"] = torch.randint(0, case["vocab"], shape, device=device, generator=gen)
        state["model"] = model = _build_model(case, seed, device)
        if case["kind"] == "eval":
            return state
        if case["lora_rank"]:
            config = lora.LoRAConfig(rank=case["lora_rank"], alpha=2.0 * case["lora_rank"],
                                     target_modules={"c_attn", "attn.c_proj"}, seed=seed % 65521 + 1)
            state["model"] = model = lora.GetLoRAModel(model, config)
            with torch.no_grad():       # an adapter that has been trained for a while: B is no longer zero
                for p in lora.GetLoRAParameters(model)[1::2]:
                    p.normal_(0.0, 0.01, generator=gen)
        trainable = [p for p in model.parameters() if p.requires_grad]
        # kept by the program like the model: a captured step goes on using the optimizer's moments
        state["optimizer"] = optimizer = Adam(trainable, 1e-4, 0.9, 0.95, 1e-8, weight_decay=0.1)
        loss_fn = CrossEntropyLoss()

        def step(x, y):
            optimizer.ZeroGrad()
            with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
                loss = loss_fn(model(x), y)
            loss.backward()
            optimizer.Step()
            return loss

        state["step"] = GraphedTrainStep(step, (state["x"], state["y"]), warmup=3) if case["graph"] else step
        # weights, gradients and moments are kept flat by the optimizer: one tensor of each
        flat = trainable[0]._itb_flat_buffer
        state["updated"] = {"weights": flat.param_buffer, "gradients": flat.grad_buffer}
        return state
    if case["kind"] == "attention":
        B, T, H, KV, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        state["qkv"] = torch.randn((B, T, (H + 2 * KV) * D), device=device, generator=gen).bfloat16().requires_grad_()
        state["dout"] = torch.randn((B, T, H * D), device=device, generator=gen).bfloat16()
        state["freqs"] = None
        if case["rope"]:
            from infinitrain_b200.nn.transformer import PrecomputeFreqsCis

            state["freqs"] = PrecomputeFreqsCis(D, max(T, 64), 500000.0, False, device)
        return state
    N, C, V = case["tokens"], case["width"], case["vocab"]
    state["x"] = torch.randn((1, N, C), device=device, generator=gen).bfloat16().requires_grad_()
    state["weight"] = torch.nn.Parameter(torch.randn((V, C), device=device, generator=gen) * 0.02)
    state["target"] = torch.randint(0, V, (1, N), device=device, generator=gen)
    return state


# --------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "train":
        loss = state["step"](state["x"], state["y"])
        return {"loss": loss.detach(), **state["updated"]}
    if case["kind"] == "eval":
        with torch.no_grad(), AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
            return state["model"](state["x"])
    if case["kind"] == "attention":
        qkv = state["qkv"]
        # RoPE rotates the projection's output in place: each pass gets a fresh one, as each layer does
        packed = qkv.clone() if case["rope"] else qkv
        out = ops.attention_packed(packed, case["heads"], case["kv_heads"], case["head_dim"], state["freqs"], 0, True)
        (dqkv,) = torch.autograd.grad(out, qkv, state["dout"])
        return out.detach(), dqkv
    with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
        loss = ops.cross_entropy(ops.linear(state["x"], state["weight"]), state["target"])
    dx, dw = torch.autograd.grad(loss, (state["x"], state["weight"]))
    return loss.detach(), dx, dw


# --------------------------------------------------------------------------- what a pass cannot do without
def _model_sizes(case):
    """(weights of one layer's matrices, of the head, of everything, attention FLOPs of one layer's forward)."""
    cfg = _config(case)
    D = cfg.head_dim()
    width, hidden = cfg.n_embd, cfg.ffn_hidden()
    gated = case["model"].startswith("llama")
    layer = width * (cfg.n_head + 2 * cfg.n_kv_head) * D + width * width + (3 if gated else 2) * width * hidden
    head = cfg.vocab_size * width
    total = cfg.n_layer * layer + head + (head if gated else cfg.block_size * width)
    attention = 2.0 * case["batch"] * cfg.n_head * D * case["seq"] * (case["seq"] + 1)
    return layer, head, total, attention


def work(case):
    if case["kind"] in ("train", "eval"):
        layer, head, total, attention = _model_sizes(case)
        tokens = case["batch"] * case["seq"]
        forward = 2.0 * tokens * (case["layers"] * layer + head) + case["layers"] * attention
        if case["kind"] == "eval":
            # bf16 weights and ids in, bf16 logits out
            return {"bytes": 2.0 * total + 8.0 * tokens + 2.0 * tokens * case["vocab"], "flops": forward}
        if case["lora_rank"]:
            cfg = _config(case)
            qkv = (cfg.n_head + 2 * cfg.n_kv_head) * cfg.head_dim()
            adapter = case["layers"] * case["lora_rank"] * (cfg.n_embd + qkv + 2 * cfg.n_embd)
            flops = 2.0 * 2.0 * tokens * (case["layers"] * layer + head) + 3.5 * case["layers"] * attention
            flops += 6.0 * tokens * adapter
            return {"bytes": 2.0 * total + 28.0 * adapter + 16.0 * tokens, "flops": flops}
        # fp32 weights and both moments read and written, gradients written
        return {"bytes": 28.0 * total + 16.0 * tokens,
                "flops": 6.0 * tokens * (case["layers"] * layer + head) + 3.5 * case["layers"] * attention}
    if case["kind"] == "attention":
        B, T, H, KV, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        forward = 2.0 * B * H * D * T * (T + 1)
        # qkv and dout in, out and dqkv out
        return {"bytes": 2.0 * B * T * D * (2 * (H + 2 * KV) + 2 * H), "flops": 3.5 * forward}
    N, C, V = case["tokens"], case["width"], case["vocab"]
    # bf16 activations in and their gradient out, fp32 weights in and their gradient out
    return {"bytes": 4.0 * N * C + 8.0 * V * C + 8.0 * N, "flops": 6.0 * N * C * V}


def tolerance(case):
    """bf16 operands and activations, fp32 accumulation.  Measured against the same pass in fp32: 2-norm errors of
    5e-3 to 9.5e-3 in the logits and gradients of whole models (largest single error 0.44), 2e-3 to 3.6e-3 for
    attention (0.22), up to 3.2e-3 for head and loss (9.4e-3)."""
    if case["kind"] in ("train", "eval"):
        return {"rel": 3e-2, "max": 0.9}
    if case["kind"] == "attention":
        return {"rel": 1.4e-2, "max": 0.9}
    return {"rel": 1.2e-2, "max": 4e-2}


# --------------------------------------------------------------------------- the same in 64 bits
def _rotate64(x, theta):
    """RoPE on interleaved pairs: x [B, T, heads, D]."""
    T, D = x.shape[1], x.shape[3]
    inv = theta ** (-torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)
    angle = torch.outer(torch.arange(T, dtype=torch.float64, device=x.device), inv)[None, :, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos()), dim=-1).flatten(-2)


def _attend64(q, k, v):
    """Causal attention of [T, heads, D] queries on [T, D] keys and values."""
    T, D = k.shape
    future = torch.ones((T, T), dtype=torch.bool, device=k.device).triu(1)
    s = torch.einsum("thd,sd->hts", q, k) * D ** -0.5
    return torch.einsum("hts,sd->thd", s.masked_fill(future, float("-inf")).softmax(-1), v)


def _attention64(qkv, heads, kv_heads, theta):
    """Self-attention on a packed projection, one key-value head of one sequence at a time (its scores are computed
    again for the backward pass)."""
    B, T, width = qkv.shape
    D = width // (heads + 2 * kv_heads)
    q, k, v = qkv.view(B, T, -1, D).split((heads, kv_heads, kv_heads), dim=2)
    if theta:
        q, k = _rotate64(q, theta), _rotate64(k, theta)
    group = heads // kv_heads
    again = torch.utils.checkpoint.checkpoint
    rows = [torch.cat([again(_attend64, q[b, :, h * group:(h + 1) * group], k[b, :, h], v[b, :, h], use_reentrant=False)
                       for h in range(kv_heads)], dim=1) for b in range(B)]
    return torch.stack(rows).flatten(2)


def _norm64(x, weight, bias, eps):
    if bias is None:
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight
    return torch.nn.functional.layer_norm(x, x.shape[-1:], weight, bias, eps)


def _logits64(cfg, weights, ids, lora_scale):
    """Logits of a GPT-2 or LLaMA-3 model; ``weights`` maps the state dict's names to 64-bit tensors."""
    F = torch.nn.functional

    def linear(x, name):
        y = F.linear(x, weights[name + ".weight"], weights.get(name + ".bias"))
        if name + ".lora_A" in weights:
            y = y + lora_scale * F.linear(F.linear(x, weights[name + ".lora_A"]), weights[name + ".lora_B"])
        return y

    def norm(x, name):
        return _norm64(x, weights[name + ".weight"], weights.get(name + ".bias"), cfg.norm_eps)

    gpt = "transformer.wpe.weight" in weights
    x = F.embedding(ids, weights["transformer.wte.weight"])
    if gpt:
        x = x + weights["transformer.wpe.weight"][:ids.shape[1]]
    for i in range(cfg.n_layer):
        h = f"transformer.h.{i}."
        qkv = linear(norm(x, h + "ln_1"), h + "attn.c_attn")
        x = x + linear(_attention64(qkv, cfg.n_head, cfg.n_kv_head, 0 if gpt else cfg.rope_theta), h + "attn.c_proj")
        y = norm(x, h + "ln_2")
        if gpt:
            y = F.gelu(linear(y, h + "mlp.c_fc"), approximate="tanh")
        else:
            y = linear(y, h + "mlp.c_fc") * F.silu(linear(y, h + "mlp.c_fc2"))
        x = x + linear(y, h + "mlp.c_proj")
    return linear(norm(x, "transformer.ln_f"), "lm_head")


def _model64(case, seed):
    if case.get("graph"):
        return None         # its state has taken warm-up steps already
    state = prepare(case, seed)
    named = state["model"].StateDict()
    leaves = {}             # by address: tied weights are one leaf
    for p in state["model"].parameters():
        leaves[p.data_ptr()] = p.detach().double().requires_grad_(case["kind"] == "train" and p.requires_grad)
    weights = {name: leaves[t.data_ptr()] for name, t in named.items() if t.data_ptr() in leaves}
    logits = _logits64(_config(case), weights, state["x"], 2.0)
    if case["kind"] == "eval":
        return logits
    loss = torch.nn.functional.cross_entropy(logits.flatten(0, 1), state["y"].flatten())
    del logits
    loss.backward()
    flat = next(p for p in state["model"].parameters() if p.requires_grad)._itb_flat_buffer
    updated, gradients = (torch.zeros(flat.param_buffer.shape, dtype=torch.float64, device=loss.device) for _ in range(2))
    for p, (begin, end, _) in zip(flat.params, flat.layout.param_ranges):
        w = leaves[p.data_ptr()]
        g = w.grad
        gradients[begin:end] = g.flatten()
        # the first AdamW step: both corrected moments are the gradient's own
        w = w.detach()
        updated[begin:end] = (w - 1e-4 * (g / (g.abs() + 1e-8) + 0.1 * w)).flatten()
    return {"loss": loss.detach(), "weights": updated, "gradients": gradients}


def exact(case, seed):
    """What ``run`` returns, by plain torch operations in 64 bits."""
    if case["kind"] in ("train", "eval"):
        return _model64(case, seed)
    state = prepare(case, seed)
    if case["kind"] == "attention":
        qkv = state["qkv"].detach().double().requires_grad_()
        out = _attention64(qkv, case["heads"], case["kv_heads"], 500000.0 if case["rope"] else 0)
        (dqkv,) = torch.autograd.grad(out, qkv, state["dout"].double())
        return out.detach(), dqkv
    x, weight = (state[k].detach().double().requires_grad_() for k in ("x", "weight"))
    loss = torch.nn.functional.cross_entropy((x @ weight.T)[0], state["target"][0])
    dx, dw = torch.autograd.grad(loss, (x, weight))
    return loss.detach(), dx, dw
