"""The work this framework is used for, as a list of measurable cases.

A case is a dict of plain values; `prepare` builds what a program holds before the call (packed weights,
scales, activations on the GPU), `run` makes one pass through the public entry points.  Activations are
bf16 N(0, 1) with 1 % of the channels twenty times larger, weights N(0, 0.02), row and column scales
log-normal(0, 0.3): the distributions of the benchmark configurations.  Layer sizes are those of
`dualquant_b200.synthetic` and of the decoder configuration, or generic ones around them.

Kinds of case:
  linear  one PermLinear.forward: 4-bit integer, MXFP4, NVFP4 or 16-bit activations against 4-bit
          weights, with or without activation scale, online Hadamard and bias
  dual    the one-call dual-scale linear with row scale and fp32 output
  mlp     the MLP block of a decoder layer: RMSNorm + gate/up, SiLU * up + Hadamard + down + residual
  prompt  Decoder.prefill on a batch of prompts
  step    one captured decode step of the decoder, replayed
  search  the offline scale search of one weight and the packing of its result
"""
import math

import torch

from dualquant_b200 import _lib, bcd, decoder, ops, quarot, wrap
from dualquant_b200.activations import PermLinear
from dualquant_b200.formats import make_format

_BLOCK = {"mxfp4": 32, "nvfp4": 16}
# input sizes of a down projection with an online Hadamard of the whole row: 28 * 2^n and its halves (the
# shards under tensor parallelism), powers of two, and 172 * 64
_FULL_HADAMARD = (1792, 3584, 7168, 14336, 2048, 4096, 8192, 11008)
_COST = 3.0e12  # multiply-adds of the largest case a draw may give


def _linear(name, tokens, k, n, act="int4", had="none", scaled=True, bias=False):
    return {"name": name, "kind": "linear", "tokens": tokens, "k": k, "n": n, "act": act, "had": had,
            "scaled": scaled, "bias": bias}


def listed():
    return [
        # the smallest call: one new token through an output projection with the Hadamard across its heads
        _linear("o_proj 1 token", 1, 4096, 4096, had="heads"),
        # a decode batch of sixteen through the widest linear of a layer: streams 59 MB of weights
        _linear("gate_up 16 tokens", 16, 4096, 28672),
        # a ragged medium batch (speculative or mixed decode) through a projection with bias
        _linear("qkv 100 tokens bias", 100, 3584, 4608, bias=True),
        # a prompt of odd length through a down projection with the online Hadamard of the whole row
        _linear("down 1531 tokens hadamard", 1531, 14336, 4096, had="full"),
        # a single dual-scale linear with row scale and fp32 output, 2048 tokens
        {"name": "dual-scale 2048 tokens fp32", "kind": "dual", "tokens": 2048, "k": 4096, "n": 4096},
        # the MLP block of one layer on a large batch of prompt tokens
        {"name": "mlp 8192 tokens", "kind": "mlp", "tokens": 8192, "hidden": 4096, "inter": 14336},
        # block-scaled FP4: a decode batch through the widest linear, a prompt through the deepest one
        _linear("mxfp4 gate_up 16 tokens", 16, 3584, 37888, act="mxfp4"),
        _linear("nvfp4 down 4096 tokens", 4096, 18944, 3584, act="nvfp4"),
        # activation quantisation switched off: 16-bit activations against the same 4-bit weights
        _linear("16-bit act 512 tokens", 512, 4096, 28672, act="none"),
        # one decode step of half a model, eight sequences with 2048 tokens of context
        {"name": "decode step 8 x 2048", "kind": "step", "batch": 8, "context": 2048, "layers": 16},
        # the prompts of the same eight sequences, four layers
        {"name": "prompts 8 x 2048", "kind": "prompt", "batch": 8, "seq": 2048, "layers": 4},
        # the offline step: scale search, block quantisation and packing of one weight
        {"name": "scale search 4096 x 4096", "kind": "search", "rows": 4096, "cols": 4096, "scale_format": "e8m0"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, step):
    """(k, n) of a linear: k a multiple of `step`, n mostly a multiple of 16, sometimes any number."""
    k = step * _log_int(rng, max(1, 1024 // step), 18944 // step)
    n = _log_int(rng, 1000, 38000)
    return k, n if rng.random() < 0.25 else (n + 15) // 16 * 16


def _tokens(rng, k, n, most=8192):
    return _log_int(rng, 1, max(2, min(most, int(_COST / k / n))))


def draw(rng):
    kind = rng.choices(("int4", "heads", "full", "fp4", "none", "dual", "mlp", "prompt", "step", "search"),
                       (6, 2, 2, 3, 1.5, 1.5, 1.5, 0.75, 0.75, 1))[0]
    if kind in ("int4", "none", "fp4"):
        act = rng.choice(("mxfp4", "nvfp4")) if kind == "fp4" else kind
        k, n = _shape(rng, 256 if kind == "fp4" else 128)
        return {"kind": "linear", "tokens": _tokens(rng, k, n), "k": k, "n": n, "act": act, "had": "none",
                "scaled": rng.random() < 0.75, "bias": rng.random() < 0.25}
    if kind in ("heads", "full"):
        k = 128 * 2 ** rng.randint(2, 5) if kind == "heads" else rng.choice(_FULL_HADAMARD)
        n = 16 * _log_int(rng, 64, 512)
        return {"kind": "linear", "tokens": _tokens(rng, k, n), "k": k, "n": n, "act": "int4", "had": kind,
                "scaled": rng.random() < 0.75, "bias": False}
    if kind == "dual":
        k, n = _shape(rng, 128)
        return {"kind": "dual", "tokens": _tokens(rng, k, n), "k": k, "n": n}
    if kind == "mlp":
        hidden, inter = 128 * _log_int(rng, 8, 40), rng.choice(_FULL_HADAMARD)
        return {"kind": "mlp", "tokens": _tokens(rng, 3 * hidden, inter), "hidden": hidden, "inter": inter}
    if kind == "prompt":
        batch = _log_int(rng, 1, 8)
        return {"kind": "prompt", "batch": batch, "seq": _log_int(rng, 16, 2048), "layers": rng.randint(1, 4)}
    if kind == "step":
        return {"kind": "step", "batch": _log_int(rng, 1, 16), "context": _log_int(rng, 64, 2048),
                "layers": rng.randint(2, 16)}
    return {"kind": "search", "rows": _log_int(rng, 512, 8192), "cols": 128 * _log_int(rng, 8, 40),
            "scale_format": rng.choice(("none", "e8m0", "e4m3"))}


# ------------------------------------------------------------------------------------------- operands
def _activations(shape, gen):
    x = torch.randn(*shape, generator=gen, device=gen.device)
    outliers = torch.randperm(shape[-1], generator=gen, device=gen.device)[: shape[-1] // 100]
    x[..., outliers] *= 20
    return x.to(torch.bfloat16)


def _weight(n, k, gen):
    return (torch.randn(n, k, generator=gen, device=gen.device) * 0.02).to(torch.bfloat16)


def _scale(n, gen):
    return torch.exp(torch.randn(n, generator=gen, device=gen.device) * 0.3).half().float()


def _on_grid(n, k, act, gen):
    """A bf16 weight as a quantised checkpoint stores it: values on the grid of its 4-bit format."""
    w = _weight(n, k, gen)
    if act in _BLOCK:
        return make_format(act, block_size=_BLOCK[act]).cast(w)
    codes, sw = ops.quant_w_int4(w)
    return (codes.view(n, k // 128, 128) * sw.float().unsqueeze(-1)).view(n, k).to(torch.bfloat16)


def _perm_linear(case, gen):
    k, n, act = case["k"], case["n"], case["act"]
    layer = torch.nn.Linear(k, n, bias=case["bias"], device="meta", dtype=torch.bfloat16)
    layer.weight = torch.nn.Parameter(_on_grid(n, k, act, gen), requires_grad=False)
    if case["bias"]:
        b = torch.randn(n, generator=gen, device=gen.device).to(torch.bfloat16)
        layer.bias = torch.nn.Parameter(b, requires_grad=False)
    fmt = make_format(act, block_size=_BLOCK[act]) if act in _BLOCK else make_format("rtn_int4", block_size=-1)
    perm = PermLinear(layer, act_fmt=fmt)
    if case["scaled"]:
        perm.set_act_scale(1.0 / _scale(k, gen))
    if case["had"] == "full":
        perm.had_K, perm.K = quarot.get_hadK(k)
        perm.online_full_had = True
    elif case["had"] == "heads":
        perm.had_K, perm.K = quarot.get_hadK(k // 128)
        perm.online_partial_had, perm.had_dim = True, 128
    if act in _BLOCK:
        perm.pack_fp4(_lib.FP4_MXFP4 if act == "mxfp4" else _lib.FP4_NVFP4, force=True)
    else:
        perm.pack()
    perm.set_act_quant_enabled(act != "none")
    return perm


def _decoder(case, gen, seed, max_len):
    cfg = decoder.DecoderConfig(num_hidden_layers=case["layers"])
    model = decoder.Decoder(cfg, gen.device, seed=seed)
    model.alloc_cache(case["batch"], max_len)
    return model


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device).manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        return {"kind": kind, "layer": _perm_linear(case, gen), "x": _activations((1, case["tokens"], case["k"]), gen)}
    if kind == "dual":
        k, n = case["k"], case["n"]
        pw = ops.pack_w_int4(*ops.quant_w_int4(_weight(n, k, gen)))
        scratch = torch.empty(ops.linear_scratch_bytes(case["tokens"], n, k), dtype=torch.uint8, device=device)
        return {"kind": kind, "pw": pw, "r": _scale(n, gen), "a": 1.0 / _scale(k, gen), "scratch": scratch,
                "x": _activations((case["tokens"], k), gen)}
    if kind == "mlp":
        hidden, inter = case["hidden"], case["inter"]
        mat, order = quarot.get_hadK(inter)
        had = ops.Hadamard(_lib.HAD_FULL, order, 0, quarot.full_hadamard_scale(inter),
                           None if mat is None else mat.to(device))
        return {"kind": kind, "inter": inter, "gate_up": decoder.W4A4Linear(2 * inter, hidden, device, gen),
                "down": decoder.W4A4Linear(hidden, inter, device, gen, had),
                "norm": torch.ones(hidden, dtype=torch.bfloat16, device=device),
                "x": _activations((case["tokens"], hidden), gen)}
    if kind == "prompt":
        model = _decoder(case, gen, seed, case["seq"])
        ids = torch.randint(0, model.cfg.vocab_size, (case["batch"], case["seq"]), generator=gen, device=device)
        return {"kind": kind, "model": model, "ids": ids}
    if kind == "step":
        model = _decoder(case, gen, seed, case["context"] + 128)
        for layer in model.layers:
            layer.k_cache[:, :, : case["context"]].normal_(generator=gen)
            layer.v_cache[:, :, : case["context"]].normal_(generator=gen)
        ids = torch.randint(0, model.cfg.vocab_size, (case["batch"],), generator=gen, device=device)
        pos = torch.tensor([case["context"]], device=device)
        with torch.no_grad():
            model.decode_step(ids, pos)  # lazy set-up happens outside the capture
            torch.cuda.synchronize(device)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                logits = model.decode_step(ids, pos)
        at = case["context"]
        new_kv = [(layer.k_cache[:, :, at], layer.v_cache[:, :, at]) for layer in model.layers]
        return {"kind": kind, "model": model, "ids": ids, "pos": pos, "graph": graph, "out": (logits, new_kv)}
    if kind == "search":
        return {"kind": kind, "scale_format": case["scale_format"],
                "w": torch.randn(case["rows"], case["cols"], generator=gen, device=device) * 0.02}
    raise ValueError(f"unknown kind of case: {kind!r}")


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "dual":
        return ops.linear_w4a4_int4(state["x"], state["a"], None, state["pw"], state["r"], scale_fp16=True,
                                    scratch=state["scratch"])
    if kind == "mlp":
        gate_up = state["gate_up"].normed(state["x"], state["norm"], 1e-5)
        return state["down"].gated(gate_up[:, : state["inter"]], gate_up[:, state["inter"]:], residual=state["x"])
    if kind == "prompt":
        model = state["model"]
        with torch.no_grad():
            logits = model.prefill(state["ids"])
        return logits, [(layer.k_cache, layer.v_cache) for layer in model.layers]
    if kind == "step":
        state["graph"].replay()
        return state["out"]
    mat_q, column_scales = bcd.dualquant_weight(state["w"], scale_format=state["scale_format"])
    packed, a = wrap.pack_from_dualquant(mat_q, column_scales)
    return mat_q, a, packed.w_packed, packed.sw_t


# ---------------------------------------------------------------------------------------- what it costs
def _linear_work(m, k, n, out_bytes, act="int4"):
    scales = n * k // _BLOCK[act] if act in _BLOCK else n * (k // 128) * 2
    return {"bytes": n * k // 2 + scales + 2 * m * k + out_bytes * m * n + 4 * k, "flops": 2 * m * n * k}


def work(case):
    kind = case["kind"]
    if kind == "linear":
        return _linear_work(case["tokens"], case["k"], case["n"], 2, case["act"])
    if kind == "dual":
        return _linear_work(case["tokens"], case["k"], case["n"], 4)
    if kind == "mlp":
        m, h, i = case["tokens"], case["hidden"], case["inter"]
        return {"bytes": 3 * h * i // 2 + 3 * h * i // 64 + 4 * m * h, "flops": 6 * m * h * i}
    if kind == "search":
        size = case["rows"] * case["cols"]
        # five rounds of two least-squares steps over the whole matrix, about eight operations an element
        return {"bytes": 8 * size + size // 2 + size // 64, "flops": 80 * size}
    cfg = decoder.DecoderConfig(num_hidden_layers=case["layers"])
    weights = decoder.linear_weight_bytes(cfg)
    per_token = weights / (0.5 + 2 / 128)
    head = cfg.vocab_size * cfg.hidden_size
    kv = 2 * cfg.num_key_value_heads * cfg.head_dim * case["layers"]
    qk = cfg.num_attention_heads * cfg.head_dim * case["layers"]
    b = case["batch"]
    if kind == "prompt":
        m = b * case["seq"]
        return {"bytes": weights + 2 * head + 2 * m * (kv + cfg.hidden_size),
                "flops": 2 * per_token * m + 2 * b * head + 2 * m * case["seq"] * qk}
    return {"bytes": weights + 2 * head + 2 * b * (case["context"] + 1) * kv + 2 * b * cfg.vocab_size,
            "flops": 2 * per_token * b + 2 * b * head + 4 * b * (case["context"] + 1) * qk}


def tolerance(case):
    kind = case["kind"]
    if kind == "dual":
        return {"rel": 1e-5}  # exact integer group sums, fp32 sums over the groups
    if kind == "linear":
        # bf16 results; behind a Hadamard the order of its fp32 sums moves codes that lie on a rounding boundary
        return {"rel": 1e-2 if case["had"] != "none" else 4e-3}
    if kind == "search":
        # fp32 sums in another order: a scale or a code at a rounding boundary may step
        return {"rel": 5e-3, "max": 0.9, "differ": 0.01}
    # several 4-bit quantisers in a row: a last-bit difference in front of one moves codes behind it
    return {"rel": 3e-2}
