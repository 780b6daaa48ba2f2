"""What this framework is timed on: the calls that its users' programs spend their time in, at the sizes of this
repository's own configurations (Llama-3.2-1B / 3B, Llama-3.1-8B, the serving sizes of the family benchmark).

Training calls a decoder layer forward and backward and the language-model head with its loss; serving calls a whole
prompt, single-token steps through captured graphs, and the mixers that the other families are built from: attention over
the cache, the sparse mixture, the recurrent mixers.  Matrix layers are single layers or blocks, so that a tolerance
belongs to one path; one listed case is a whole model, one half of one.

``prepare`` makes inputs from the seed alone; ``exact`` restates every path in float64 with plain torch.
"""
import math

import torch
import torch.nn.functional as F

# hidden, intermediate, query heads, key/value heads, head size
LLAMA = {"1b": (2048, 8192, 32, 8, 64), "3b": (3072, 8192, 24, 8, 128), "8b": (4096, 14336, 32, 8, 128)}
LLAMA_VOCAB = 128256
EPS = 1e-5
THETA = 500000.0


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def listed():
    return [
        # one layer of the headline training step: 3B, one sequence of 8192 tokens, forward and backward
        {"name": "train_layer_3b_8k", "kind": "train_layer", "size": "3b", "batch": 1, "seq": 8192},
        # the 1B layer on a batch that is no multiple of any tile: the last batch of an epoch, variable-length fine-tuning
        {"name": "train_layer_1b_ragged", "kind": "train_layer", "size": "1b", "batch": 2, "seq": 1531},
        # final norm, output head over the whole vocabulary and the loss, forward and backward
        {"name": "loss_head_3b", "kind": "loss_head", "hidden": 3072, "vocab": LLAMA_VOCAB, "tokens": 4001},
        # time to first token: half of a 1B model and the head on one prompt, called as a program without graphs does
        {"name": "prompt_1b", "kind": "prompt", "size": "1b", "layers": 8, "batch": 1, "seq": 2048},
        # one token of one user: a whole 1B model through its captured graph, the latency-bound end of serving
        {"name": "token_1b", "kind": "token", "size": "1b", "layers": 16, "batch": 1, "context": 2048},
        # one token of many users with contexts of many lengths: a stage of four 1B layers and the head
        {"name": "token_1b_batch", "kind": "token", "size": "1b", "layers": 4, "batch": 64, "context": 2048},
        # attention of single tokens over a paged cache, a handful of users with contexts of many lengths
        {"name": "paged_attention", "kind": "token_attention", "size": "3b", "batch": 12, "context": 2900, "paged": True},
        # a portion of a long prompt on top of what the cache holds already, sliding window, kept first tokens, distance
        # bias
        {"name": "window_portion", "kind": "window_portion", "heads": 32, "kv_heads": 8, "dim": 128, "batch": 2,
         "portion": 2048, "past": 2048, "window": 2048, "keep": 4, "bias": True},
        # sparse feed-forward of a prompt batch: every expert gets many tokens
        {"name": "experts_prompt", "kind": "experts", "width": 2048, "experts": 8, "top": 2, "ff": 2048, "tokens": 8190,
         "dtype": "bf16"},
        # sparse feed-forward of a token step: the tokens of a small batch meet most of the experts
        {"name": "experts_token", "kind": "experts", "width": 1024, "experts": 16, "top": 4, "ff": 512, "tokens": 64,
         "dtype": "bf16"},
        # a prompt batch through the gated delta rule: short convolution, unit norms, recurrence
        {"name": "delta_prompt", "kind": "delta_prompt", "heads": 4, "kv_heads": 4, "dim": 128, "vdim": 256, "batch": 4,
         "seq": 2048, "channel": False},
        # a prompt batch through retention in fp32, the type of the families' accuracy replays
        {"name": "retention_prompt_fp32", "kind": "retention_prompt", "heads": 8, "dim": 256, "vdim": 512, "batch": 2,
         "seq": 4096, "dtype": "fp32"},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["train_layer", "loss_head", "prompt", "token", "token_attention", "window_portion", "experts",
                       "delta_prompt", "retention_prompt"])
    if kind == "train_layer":
        size = rng.choice(["1b", "3b", "8b"])
        batch = rng.choice([1, 2, 3])
        return {"kind": kind, "size": size, "batch": batch,
                "seq": max(33, _log(rng, 128, 2048 if size == "8b" else 7000) // batch)}
    if kind == "loss_head":
        return {"kind": kind, "hidden": rng.choice([2048, 3072]), "vocab": rng.choice([32000, LLAMA_VOCAB]),
                "tokens": _log(rng, 64, 4096)}
    if kind == "prompt":
        return {"kind": kind, "size": rng.choice(["1b", "3b"]), "layers": rng.randint(2, 6), "batch": rng.choice([1, 2, 4]),
                "seq": _log(rng, 64, 2048)}
    if kind == "token":
        return {"kind": kind, "size": rng.choice(["1b", "3b"]), "layers": rng.randint(2, 6), "batch": _log(rng, 1, 80),
                "context": _log(rng, 100, 3000)}
    if kind == "token_attention":
        return {"kind": kind, "size": rng.choice(["1b", "3b", "8b"]), "batch": _log(rng, 1, 64),
                "context": _log(rng, 64, 8000), "paged": rng.random() < 0.5}
    if kind == "window_portion":
        heads, kv_heads, dim = rng.choice([(16, 4, 128), (32, 8, 128), (16, 16, 64), (16, 4, 64)])
        return {"kind": kind, "heads": heads, "kv_heads": kv_heads, "dim": dim, "batch": rng.choice([1, 2, 3]),
                "portion": _log(rng, 64, 2100), "past": rng.randint(1, 3000), "window": rng.choice([512, 1024, 2048]),
                "keep": rng.choice([0, 4]), "bias": rng.random() < 0.5}
    if kind == "experts":
        width, experts, top, ff = rng.choice([(2048, 8, 2, 2048), (4096, 8, 2, 4096), (1024, 16, 4, 512)])
        dtype = "bf16" if rng.random() < 0.75 else "fp32"
        return {"kind": kind, "width": width, "experts": experts, "top": top, "ff": ff, "dtype": dtype,
                "tokens": _log(rng, 1, 8192 if dtype == "bf16" else 300)}
    if kind == "delta_prompt":
        heads, dim, vdim = rng.choice([(4, 128, 256), (8, 256, 512), (4, 64, 128)])
        batch = rng.choice([1, 2, 4])
        return {"kind": kind, "heads": heads, "kv_heads": rng.choice([heads, heads // 2]), "dim": dim, "vdim": vdim,
                "batch": batch, "seq": _log(rng, 70, 4096) // (2 if batch == 4 else 1), "channel": rng.random() < 0.4}
    heads, dim, vdim = rng.choice([(4, 128, 256), (8, 256, 512), (4, 64, 128)])
    batch = rng.choice([1, 2, 4])
    return {"kind": kind, "heads": heads, "dim": dim, "vdim": vdim, "batch": batch,
            "seq": max(64, _log(rng, 70, 4096) // (2 if batch == 4 else 1)), "dtype": rng.choice(["bf16", "fp32"])}


# ---- inputs ----------------------------------------------------------------------------------------------------------------


class _Draws:
    def __init__(self, seed):
        self.g = torch.Generator(device=_device()).manual_seed(int(seed) % (1 << 62))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.empty(shape, dtype=dtype, device=_device())
        return t.normal_(mean, std, generator=self.g)

    def ints(self, low, high, shape):
        return torch.randint(low, high, shape, generator=self.g, device=_device())


def _dtype(case):
    return torch.float32 if case.get("dtype") == "fp32" else torch.bfloat16


def _layer_weights(d, size, prefix=""):
    H, I, nq, nkv, D = LLAMA[size]
    return {prefix + "self_attn.qkv_proj.weight_qkv": d.normal((nq + 2 * nkv) * D, H, std=0.02),
            prefix + "self_attn.o_proj.weight": d.normal(H, nq * D, std=0.02),
            prefix + "mlp.gate_up_proj.weight": d.normal(2 * I, H, std=0.02),
            prefix + "mlp.down_proj.weight": d.normal(H, I, std=0.02),
            prefix + "input_layernorm.weight": d.normal(H, std=0.1, mean=1.0),
            prefix + "post_attention_layernorm.weight": d.normal(H, std=0.1, mean=1.0)}


def _model_weights(d, case):
    H = LLAMA[case["size"]][0]
    w = {"model.embed_tokens.weight": d.normal(LLAMA_VOCAB, H, std=0.02), "model.norm.weight": d.normal(H, std=0.1, mean=1.0)}
    for i in range(case["layers"]):
        w.update(_layer_weights(d, case["size"], "model.layers.%d." % i))
    return w


def _lengths(d, case):
    """Tokens per sequence, the new one counted: all of the context for one sequence, else spread over its upper half
    and more, one row at the full length."""
    n, B = case["context"], case["batch"]
    if B == 1:
        return torch.full((1,), n, dtype=torch.long, device=_device())
    lens = d.ints(max(1, n // 3), n + 1, (B,))
    lens[0] = n
    return lens


def _inputs(case, seed):
    d, kind = _Draws(seed), case["kind"]
    if kind == "train_layer":
        H, S, B = LLAMA[case["size"]][0], case["seq"], case["batch"]
        return {"w": _layer_weights(d, case["size"]), "hidden": d.normal(S, B, H, std=0.5), "residual": d.normal(S, B, H),
                "d_hidden": d.normal(S, B, H, std=0.1), "d_residual": d.normal(S, B, H, std=0.1)}
    if kind == "loss_head":
        N, H, V = case["tokens"], case["hidden"], case["vocab"]
        return {"norm": d.normal(H, std=0.1, mean=1.0), "head": d.normal(V, H, std=0.02), "hidden": d.normal(N, 1, H, std=0.5),
                "residual": d.normal(N, 1, H), "labels": d.ints(0, V, (1, N))}
    if kind == "prompt":
        return {"w": _model_weights(d, case), "ids": d.ints(0, LLAMA_VOCAB, (case["batch"], case["seq"]))}
    if kind == "token":
        H, I, nq, nkv, D = LLAMA[case["size"]]
        S = (case["context"] + 255) // 256 * 256
        shape = (case["batch"], nkv, S, D)
        return {"w": _model_weights(d, case), "ids": d.ints(0, LLAMA_VOCAB, (case["batch"], 1)), "lens": _lengths(d, case),
                "k": [d.normal(*shape) for _ in range(case["layers"])], "v": [d.normal(*shape) for _ in range(case["layers"])]}
    if kind == "token_attention":
        H, I, nq, nkv, D = LLAMA[case["size"]]
        B, page = case["batch"], 128
        pages = (case["context"] + page - 1) // page
        x = {"q": d.normal(B, nq, D), "lens": _lengths(d, case)}
        shape = (B * pages, nkv, page, D) if case["paged"] else (B, nkv, pages * page, D)
        x["k"], x["v"] = d.normal(*shape), d.normal(*shape)
        if case["paged"]:
            x["table"] = torch.randperm(B * pages, generator=d.g, device=_device()).to(torch.int32).reshape(B, pages)
        return x
    if kind == "window_portion":
        B, T, H, G, D = case["batch"], case["portion"], case["heads"], case["kv_heads"], case["dim"]
        S = (case["past"] + T + 127) // 128 * 128
        h = torch.arange(1, H + 1, dtype=torch.float64)
        return {"q": d.normal(B, T, H, D), "k": d.normal(B, G, S, D), "v": d.normal(B, G, S, D),
                "slopes": torch.pow(2.0, -8.0 * h / H).to(torch.float32).to(_device()) if case["bias"] else None,
                "start": torch.full((B,), case["past"], dtype=torch.int32, device=_device())}
    if kind == "experts":
        W, E, f, dt = case["width"], case["experts"], case["ff"], _dtype(case)
        return {"router": d.normal(E, W, std=W ** -0.5, dtype=torch.float32),
                "correction": d.normal(E, std=0.01, dtype=torch.float32),
                "gate_up": d.normal(E, W, 2 * f, std=0.02, dtype=dt), "down": d.normal(E, f, W, std=0.02, dtype=dt),
                "h": d.normal(case["tokens"], W, dtype=dt)}
    if kind == "delta_prompt":
        B, T, H, G, D, Dv = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "dim", "vdim"))
        C, na = 2 * G * D + H * Dv, H * D if case["channel"] else H
        return {"proj": d.normal(B, T, C), "conv_w": d.normal(C, 4, std=0.5, dtype=torch.float32),
                "conv": d.normal(B, 3, C, dtype=torch.float32), "S": d.normal(B, H, D, Dv, dtype=torch.float32),
                "a_pre": d.normal(B * T, na, dtype=torch.float32), "b_pre": d.normal(B * T, H, dtype=torch.float32),
                "a_log": d.normal(H, std=0.5, mean=-2.0, dtype=torch.float32), "dt_bias": d.normal(na, dtype=torch.float32),
                "start": torch.zeros(B, dtype=torch.int32, device=_device())}
    B, T, H, D, Dv = (case[k] for k in ("batch", "seq", "heads", "dim", "vdim"))
    half = torch.arange(D // 2, dtype=torch.float64)
    ang = torch.outer(torch.arange(T, dtype=torch.float64), torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2.0 * half / D))
    steps = torch.linspace(math.log(1 / 32), math.log(1 / 512), H, dtype=torch.float64)
    return {"proj": d.normal(B, T, 2 * H * D + H * Dv, dtype=_dtype(case)), "S": d.normal(B, H, D, Dv, dtype=torch.float32),
            "cos": ang.cos().float().to(_device()), "sin": ang.sin().float().to(_device()),
            "decay": (1 - steps.exp()).float().to(_device()), "start": torch.zeros(B, dtype=torch.int32, device=_device())}


def _config(case, **kw):
    from neuronx_distributed_llama3_2_b200.models import llama

    make = {"1b": llama.llama3_2_1b, "3b": llama.llama3_2_3b, "8b": llama.llama3_1_8b}[case["size"]]
    return make(rope_scaling=None, **kw)


def _fill(module, weights):
    own = dict(module.named_parameters())
    with torch.no_grad():
        for name, w in weights.items():
            own[name].copy_(w)


# ---- the state that a program keeps, and one pass ----------------------------------------------------------------------------


def prepare(case, seed):
    kind, dev = case["kind"], _device()
    x = _inputs(case, seed)
    if kind == "train_layer":
        from neuronx_distributed_llama3_2_b200.models.llama import LlamaDecoderLayer
        from neuronx_distributed_llama3_2_b200.ops.rope import build_rope_cache

        cfg = _config(case)
        layer = LlamaDecoderLayer(cfg, device=dev).train()
        _fill(layer, x.pop("w"))
        cos, sin = build_rope_cache(case["seq"], cfg.head_dim, cfg.rope_theta, None, device=dev)
        return {"kind": kind, "layer": layer, "cos": cos, "sin": sin, **x}
    if kind == "loss_head":
        from neuronx_distributed_llama3_2_b200.models.llama import CausalLMLoss
        from neuronx_distributed_llama3_2_b200.parallel.layer_norm import RMSNorm
        from neuronx_distributed_llama3_2_b200.parallel.layers import ColumnParallelLinear

        norm = RMSNorm(case["hidden"], EPS, sequence_parallel_enabled=True, dtype=torch.bfloat16, device=dev)
        head = ColumnParallelLinear(case["hidden"], case["vocab"], bias=False, gather_output=False,
                                    sequence_parallel_enabled=True, dtype=torch.bfloat16, device=dev)
        _fill(norm, {"weight": x.pop("norm")})
        _fill(head, {"weight": x.pop("head")})
        return {"kind": kind, "norm": norm, "head": head, "loss": CausalLMLoss(), **x}
    if kind in ("prompt", "token"):
        from neuronx_distributed_llama3_2_b200.inference.config import InferenceConfig
        from neuronx_distributed_llama3_2_b200.inference.model import LlamaInferenceModel
        from neuronx_distributed_llama3_2_b200.inference.model_builder import BaseModelInstance, ModelBuilder

        class LogitsModel(LlamaInferenceModel):
            """The graph of a program that samples on its own: the step's logits come back."""

            def forward(self, input_ids, position_ids, seq_ids=None, last_token_index=None):
                return self.forward_infer(input_ids, position_ids, seq_ids, last_token_index, return_logits=True,
                                          sample=False)[1]

        B = case["batch"]
        T = case["seq"] if kind == "prompt" else 1
        S = case["seq"] if kind == "prompt" else x["k"][0].shape[2]
        model = LogitsModel(_config(case, num_hidden_layers=case["layers"]),
                            InferenceConfig(batch_size=B, max_context_length=S, seq_len=S), device=dev)
        _fill(model, x.pop("w"))
        cache = model.init_kv_cache(device=dev)
        pos = (torch.arange(T, device=dev).unsqueeze(0).expand(B, T).contiguous() if kind == "prompt"
               else (x["lens"] - 1).reshape(B, 1))
        args = (x["ids"], pos, torch.arange(B, dtype=torch.int32, device=dev),
                torch.full((B,), T - 1, dtype=torch.long, device=dev))
        if kind == "prompt":
            return {"kind": kind, "call": model, "args": args, "cache": cache}
        for mine, given in zip(cache.k + cache.v, x["k"] + x["v"]):
            mine.copy_(given)
        builder = ModelBuilder(use_cuda_graphs=dev.type == "cuda")
        builder.add("token_generation_model", BaseModelInstance(lambda: model), [args])
        return {"kind": kind, "call": builder.trace(initialize_model_weights=False), "args": args, "cache": cache}
    if kind == "experts":
        from neuronx_distributed_llama3_2_b200.modules.moe.sparse import SparseMoE

        block = SparseMoE(case["width"], case["experts"], case["top"], case["ff"], 7.0, dtype=_dtype(case), device=dev).eval()
        _fill(block, {"router.linear_router.weight": x["router"], "router.correction": x["correction"],
                      "experts.gate_up_proj.weight": x["gate_up"], "experts.down_proj.weight": x["down"]})
        return {"kind": kind, "block": block, "h": x["h"]}
    return {"kind": kind, "case": dict(case), **x}


def run(state):
    kind, s = state["kind"], state
    if kind == "train_layer":
        layer = s["layer"]
        layer.zero_grad(set_to_none=True)
        hidden, residual = (s[k].detach().requires_grad_() for k in ("hidden", "residual"))
        out = layer(hidden, residual, s["cos"], s["sin"])
        torch.autograd.backward(out, (s["d_hidden"], s["d_residual"]))
        return {"out": out[0].detach(), "stream": out[1].detach(), "d_hidden": hidden.grad, "d_residual": residual.grad,
                "grads": {n: p.grad for n, p in layer.named_parameters()}}
    if kind == "loss_head":
        s["norm"].zero_grad(set_to_none=True)
        s["head"].zero_grad(set_to_none=True)
        hidden, residual = (s[k].detach().requires_grad_() for k in ("hidden", "residual"))
        loss = s["loss"](s["head"](s["norm"](hidden, residual)), s["labels"])
        loss.backward()
        return {"loss": loss.detach(), "d_hidden": hidden.grad, "d_residual": residual.grad, "d_norm": s["norm"].weight.grad,
                "d_head": s["head"].weight.grad}
    if kind in ("prompt", "token"):
        with torch.no_grad():
            return {"logits": s["call"](*s["args"]), "k": list(s["cache"].k), "v": list(s["cache"].v)}
    if kind == "token_attention":
        from neuronx_distributed_llama3_2_b200.ops.attention import decode_attention

        return decode_attention(s["q"], s["k"], s["v"], s["lens"], block_table=s.get("table"),
                                page_size=128 if "table" in s else 0)
    if kind == "window_portion":
        from neuronx_distributed_llama3_2_b200.ops.window_attention import window_attention_prefill

        c = s["case"]
        return window_attention_prefill(s["q"], s["k"], s["v"], s["start"], c["dim"] ** -0.5, c["window"], c["keep"],
                                        s["slopes"])
    if kind == "experts":
        with torch.no_grad():
            return s["block"](s["h"])
    c = s["case"]
    if kind == "delta_prompt":
        from neuronx_distributed_llama3_2_b200.ops.delta_rule import delta_prep, delta_scan

        H, G, D, Dv = c["heads"], c["kv_heads"], c["dim"], c["vdim"]
        q, k, v = delta_prep(s["proj"], (0, G * D, 2 * G * D), s["conv_w"], s["conv"], s["start"], H, G, D, Dv, D ** -0.5)
        # the scan takes the gates' pre-activations over, fresh from the step's projection
        out = delta_scan(q, k, v, s["a_pre"].clone(), 0, s["b_pre"].clone(), 0, s["a_log"], s["dt_bias"], s["S"], s["start"],
                         c["channel"])
        return {"out": out, "S": s["S"], "conv": s["conv"]}
    from neuronx_distributed_llama3_2_b200.ops.retention import retention_chunkwise

    H, D, Dv = c["heads"], c["dim"], c["vdim"]
    out = retention_chunkwise(s["proj"], (0, H * D, 2 * H * D), s["decay"], s["S"], s["start"], H, D, Dv, D ** -0.5,
                              (s["cos"], s["sin"]))
    return {"out": out, "S": s["S"]}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------


def _layer_numbers(size):
    H, I, nq, nkv, D = LLAMA[size]
    return H * (nq + 2 * nkv) * D + H * nq * D + 3 * H * I


def work(case):
    kind = case["kind"]
    if kind == "train_layer":
        H, I, nq, nkv, D = LLAMA[case["size"]]
        N, n = case["batch"] * case["seq"], _layer_numbers(case["size"])
        attention = 4 * case["batch"] * nq * D * case["seq"] * (case["seq"] + 1) / 2
        return {"bytes": 2 * (2 * n + 8 * N * H), "flops": 3 * (2 * N * n + attention)}
    if kind == "loss_head":
        N, n = case["tokens"], case["hidden"] * case["vocab"]
        return {"bytes": 2 * (2 * n + 4 * N * case["hidden"]), "flops": 6 * N * n}
    if kind in ("prompt", "token"):
        H, I, nq, nkv, D = LLAMA[case["size"]]
        n, head, B = case["layers"] * _layer_numbers(case["size"]), H * LLAMA_VOCAB, case["batch"]
        if kind == "prompt":
            N = B * case["seq"]
            pairs = B * case["seq"] * (case["seq"] + 1) / 2
            return {"bytes": 2 * (n + head + N * H + case["layers"] * 2 * N * nkv * D + B * LLAMA_VOCAB),
                    "flops": 2 * N * n + 2 * B * head + 4 * pairs * nq * D * case["layers"]}
        keys = case["context"] if B == 1 else B * case["context"] * 2 / 3
        return {"bytes": 2 * (n + head + case["layers"] * 2 * keys * nkv * D + B * LLAMA_VOCAB),
                "flops": 2 * B * (n + head) + 4 * keys * nq * D * case["layers"]}
    if kind == "token_attention":
        H, I, nq, nkv, D = LLAMA[case["size"]]
        B = case["batch"]
        keys = case["context"] if B == 1 else B * case["context"] * 2 / 3
        return {"bytes": 2 * (2 * keys * nkv * D + 2 * B * nq * D), "flops": 4 * keys * nq * D}
    if kind == "window_portion":
        B, T, H, G, D = case["batch"], case["portion"], case["heads"], case["kv_heads"], case["dim"]
        pairs = sum(min(case["past"] + t + 1, case["window"] + max(0, min(case["keep"], case["past"] + t + 1 - case["window"])))
                    for t in range(T))
        rows = min(case["past"] + T, case["window"] + T + case["keep"])
        return {"bytes": 2 * B * (2 * T * H * D + 2 * rows * G * D), "flops": 4 * B * H * D * pairs}
    if kind == "experts":
        W, E, f, N, top = (case[k] for k in ("width", "experts", "ff", "tokens", "top"))
        size = 4 if case["dtype"] == "fp32" else 2
        met = E * (1 - (1 - top / E) ** N)
        return {"bytes": size * (met * 3 * W * f + N * W) + 4 * N * W, "flops": 2 * N * top * 3 * W * f}
    if kind == "delta_prompt":
        B, T, H, G, D, Dv = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "dim", "vdim"))
        C, na = 2 * G * D + H * Dv, H * D if case["channel"] else H
        return {"bytes": B * T * (2 * C + 4 * (na + H) + 4 * H * Dv) + 4 * B * H * D * Dv,
                "flops": B * T * (8 * C + 6 * H * D * Dv)}
    B, T, H, D, Dv = (case[k] for k in ("batch", "seq", "heads", "dim", "vdim"))
    size = 4 if case["dtype"] == "fp32" else 2
    return {"bytes": B * T * H * (size * (2 * D + Dv) + 4 * Dv) + 4 * B * H * D * Dv, "flops": 4 * B * T * H * D * Dv}


def tolerance(case):
    kind = case["kind"]
    if kind in ("train_layer", "prompt", "token"):      # several roundings to bf16 follow one another
        return {"rel": 3e-2}
    if kind in ("loss_head", "token_attention", "window_portion"):
        return {"rel": 1e-2}
    if kind == "experts":
        return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1e-5}
    return {"rel": 1e-5}


# ---- the same in float64 ---------------------------------------------------------------------------------------------------------


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _angles(pos, dim, base):
    freq = torch.pow(torch.tensor(float(base), dtype=torch.float64, device=pos.device),
                     -torch.arange(0, dim, 2, dtype=torch.float64, device=pos.device) / dim)
    a = pos.double().unsqueeze(-1) * freq
    return a.cos(), a.sin()


def _turn(x, cos, sin):
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _head(q, k, v):
    """One head: q, k, v [T, D], causal."""
    s = (q @ k.t()) * q.shape[-1] ** -0.5
    return torch.softmax(s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), -math.inf), dim=-1) @ v


def _causal(q, k, v):
    """q [B, T, nq, D], k and v [B, T, nkv, D]: head by head, each recomputed in its backward."""
    from torch.utils.checkpoint import checkpoint

    g = q.shape[2] // k.shape[2]
    rows = []
    for b in range(q.shape[0]):
        heads = []
        for h in range(q.shape[2]):
            args = (q[b, :, h], k[b, :, h // g], v[b, :, h // g])
            heads.append(checkpoint(_head, *args, use_reentrant=False) if torch.is_grad_enabled() else _head(*args))
        rows.append(torch.stack(heads, dim=1))
    return torch.stack(rows)


def _layer64(w, p, size, x, attend):
    """x [B, T, H] -> the feed-forward's output and the stream it is added to."""
    H, I, nq, nkv, D = LLAMA[size]
    qkv = _rms(x, w[p + "input_layernorm.weight"]) @ w[p + "self_attn.qkv_proj.weight_qkv"].t()
    x = x + attend(*qkv.unflatten(-1, (nq + 2 * nkv, D)).split([nq, nkv, nkv], dim=2)).flatten(2) \
        @ w[p + "self_attn.o_proj.weight"].t()
    gate, up = (_rms(x, w[p + "post_attention_layernorm.weight"]) @ w[p + "mlp.gate_up_proj.weight"].t()).chunk(2, dim=-1)
    return (F.silu(gate) * up) @ w[p + "mlp.down_proj.weight"].t(), x


def _exact_train_layer(case, x):
    w = {k: t.double().requires_grad_() for k, t in x["w"].items()}
    hidden, residual = (x[k].double().requires_grad_() for k in ("hidden", "residual"))
    cos, sin = (t.unsqueeze(1) for t in _angles(torch.arange(case["seq"], device=_device()), LLAMA[case["size"]][4], THETA))

    def attend(q, k, v):
        return _causal(_turn(q, cos, sin), _turn(k, cos, sin), v)

    out, stream = (t.transpose(0, 1) for t in _layer64(w, "", case["size"], (hidden + residual).transpose(0, 1), attend))
    torch.autograd.backward((out, stream), (x["d_hidden"].double(), x["d_residual"].double()))
    return {"out": out.detach(), "stream": stream.detach(), "d_hidden": hidden.grad, "d_residual": residual.grad,
            "grads": {k: t.grad for k, t in w.items()}}


def _exact_loss_head(case, x):
    norm, head, hidden, residual = (x[k].double().requires_grad_() for k in ("norm", "head", "hidden", "residual"))
    logits = _rms(hidden + residual, norm)[:, 0] @ head.t()
    loss = F.cross_entropy(logits[:-1], x["labels"][0, 1:])
    loss.backward()
    return {"loss": loss.detach(), "d_hidden": hidden.grad, "d_residual": residual.grad, "d_norm": norm.grad, "d_head": head.grad}


def _exact_model(case, x):
    H, I, nq, nkv, D = LLAMA[case["size"]]
    w, prompt = x["w"], case["kind"] == "prompt"
    B, T = x["ids"].shape
    pos = torch.arange(T, device=_device()).expand(B, T) if prompt else (x["lens"] - 1).reshape(B, 1)
    cos, sin = (t.unsqueeze(2) for t in _angles(pos, D, THETA))
    stream = w["model.embed_tokens.weight"][x["ids"]].double()
    keys, values = [], []
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        w64 = {k: t.double() for k, t in w.items() if k.startswith(p)}

        def attend(q, k, v):
            q, k = _turn(q, cos, sin), _turn(k, cos, sin)
            if prompt:
                keys.append(k.transpose(1, 2))
                values.append(v.transpose(1, 2))
                return _causal(q, k, v)
            ck, cv = x["k"][i].double(), x["v"][i].double()
            for b in range(B):
                ck[b, :, int(pos[b, 0])], cv[b, :, int(pos[b, 0])] = k[b, 0], v[b, 0]
            keys.append(ck)
            values.append(cv)
            return _over_cache(q[:, 0], ck, cv, x["lens"]).unsqueeze(1)

        out, stream = _layer64(w64, p, case["size"], stream, attend)
        stream = stream + out
    logits = _rms(stream[:, -1], w["model.norm.weight"].double()) @ w["model.embed_tokens.weight"].double().t()
    return {"logits": logits, "k": keys, "v": values}


def _over_cache(q, k, v, lens):
    """q [B, nq, D] over k and v [B, nkv, S, D], the first lens[b] rows of each."""
    g = q.shape[1] // k.shape[1]
    rows = []
    for b in range(q.shape[0]):
        n = int(lens[b])
        kb, vb = (t[b, :, :n].double() for t in (k, v))
        s = torch.einsum("ghd,gnd->ghn", q[b].double().unflatten(0, (-1, g)), kb) * q.shape[-1] ** -0.5
        rows.append(torch.einsum("ghn,gnd->ghd", torch.softmax(s, dim=-1), vb).flatten(0, 1))
    return torch.stack(rows)


def _exact_token_attention(case, x):
    k, v = x["k"], x["v"]
    if case["paged"]:
        k, v = (t[x["table"].long()].transpose(1, 2).flatten(2, 3) for t in (k, v))
    return _over_cache(x["q"], k, v, x["lens"])


def _exact_window_portion(case, x):
    H, G = case["heads"], case["kv_heads"]
    n = case["past"] + case["portion"]
    i = torch.arange(case["past"], n, device=_device()).unsqueeze(1)
    j = torch.arange(n, device=_device()).unsqueeze(0)
    hidden = ~((j <= i) & ((i - j < case["window"]) | (j < case["keep"])))
    out = torch.empty(x["q"].shape, dtype=torch.float64, device=_device())
    for b in range(case["batch"]):
        for h in range(H):
            k, v = (x[c][b, h // (H // G), :n].double() for c in ("k", "v"))
            s = x["q"][b, :, h].double() @ k.t() * case["dim"] ** -0.5
            if x["slopes"] is not None:
                s = s - x["slopes"][h].double() * (i - j)
            out[b, :, h] = torch.softmax(s.masked_fill(hidden, -math.inf), dim=-1) @ v
    return out


def _exact_experts(case, x):
    h = x["h"].double()
    score = torch.softmax(h @ x["router"].double().t(), dim=-1)
    chosen = torch.topk(score + x["correction"].double(), case["top"], dim=-1).indices
    y = torch.zeros_like(h)
    for e in range(case["experts"]):
        rows = (chosen == e).any(-1).nonzero()[:, 0]
        gate, up = (h[rows] @ x["gate_up"][e].double()).chunk(2, dim=-1)
        gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
        y[rows] += score[rows, e:e + 1] * ((gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ x["down"][e].double())
    return y


def _exact_delta_prompt(case, x):
    B, T, H, G, D, Dv = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "dim", "vdim"))
    raw = torch.cat([torch.zeros(B, 3, x["proj"].shape[2], dtype=torch.float64, device=_device()), x["proj"].double()], dim=1)
    act = F.silu(sum(x["conv_w"][:, j].double() * raw[:, j:j + T] for j in range(4)))
    q, k, v = act.split([G * D, G * D, H * Dv], dim=-1)
    q, k = (t.unflatten(-1, (G, D)) for t in (q, k))
    q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(H // G, dim=2) for t in (q * D ** -0.5, k))
    v = v.unflatten(-1, (H, Dv))
    pre = (x["a_pre"].double() + x["dt_bias"].double()).reshape(B, T, H, -1)
    g = torch.exp(-torch.exp(x["a_log"].double()).reshape(H, 1) * F.softplus(pre))
    beta = torch.sigmoid(x["b_pre"].double()).reshape(B, T, H, 1)
    S = torch.zeros(B, H, D, Dv, dtype=torch.float64, device=_device())
    out = torch.empty(B, T, H, Dv, dtype=torch.float64, device=_device())
    for t in range(T):
        S = S * g[:, t].unsqueeze(-1)
        u = beta[:, t] * (v[:, t] - (k[:, t].unsqueeze(-2) @ S).squeeze(-2))
        S = S + k[:, t].unsqueeze(-1) * u.unsqueeze(-2)
        out[:, t] = (q[:, t].unsqueeze(-2) @ S).squeeze(-2)
    return {"out": out, "S": S, "conv": raw[:, -3:]}


def _exact_retention_prompt(case, x):
    B, T, H, D, Dv = (case[k] for k in ("batch", "seq", "heads", "dim", "vdim"))
    q, k, v = x["proj"].double().split([H * D, H * D, H * Dv], dim=-1)
    cos, sin = (x[c].double().unsqueeze(1) for c in ("cos", "sin"))
    q, k = (_turn(t.unflatten(-1, (H, D)), cos, sin) for t in (q, k))
    v = v.unflatten(-1, (H, Dv))
    k = k * D ** -0.5
    t = torch.arange(T, dtype=torch.float64, device=_device())
    out, S = torch.empty_like(v), torch.empty(B, H, D, Dv, dtype=torch.float64, device=_device())
    for h in range(H):
        a = x["decay"][h].double()
        fade = torch.pow(a, (t.unsqueeze(1) - t).clamp(min=0)).tril()
        for b in range(B):
            out[b, :, h] = (q[b, :, h] @ k[b, :, h].t() * fade) @ v[b, :, h]
            S[b, h] = (k[b, :, h] * torch.pow(a, T - 1 - t).unsqueeze(1)).t() @ v[b, :, h]
    return {"out": out, "S": S}


def exact(case, seed):
    x = _inputs(case, seed)
    by_kind = {"train_layer": _exact_train_layer, "loss_head": _exact_loss_head, "prompt": _exact_model, "token": _exact_model,
               "token_attention": _exact_token_attention, "window_portion": _exact_window_portion, "experts": _exact_experts,
               "delta_prompt": _exact_delta_prompt, "retention_prompt": _exact_retention_prompt}
    if case["kind"] in ("train_layer", "loss_head"):
        return by_kind[case["kind"]](case, x)
    with torch.no_grad():
        return by_kind[case["kind"]](case, x)
