"""The work this framework is used for, as cases whose time and results can be compared between two states of the code.

A case goes through the public entry points only: `sbvr.linear`, `sbvr.mm_T`, `sbvr.row_deq_mm_T`, `sbvr.sbvr(...)` (the
encoder), `.decode()`, and the model's `generate`, `prefill` and `forward`.  Weights are random packed tensors in the
reference's layout with the value distributions the tests and the benchmark use; nothing is read from disk.
"""
import math
import os
import sys

import torch

PKG = os.path.join(os.getcwd(), "sbvr-cpu-arm_b200")      # the package's folder name is not an importable name
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import sbvr  # noqa: E402
from models.sbvr_llama import LlamaConfig, SBVRLlamaForCausalLM  # noqa: E402

# Decoder shapes of this repository's presets: hidden, intermediate, query heads, KV heads, vocabulary, codebook lines.
SHAPES = {
    "tiny8": (2048, 4096, 16, 8, 1024, 256),
    "8b": (4096, 14336, 32, 8, 128256, 4096),
    "70b": (8192, 28672, 64, 8, 128256, 4096),
}


def listed():
    return [
        # One small projection (k or v of the 8B preset) on one token: the shortest call there is, latency only.
        {"name": "linear_kv_m1", "kind": "linear", "M": 1, "N": 1024, "K": 4096, "S": 4, "G": 256, "form": "u16",
         "bias": False},
        # The seven linears of an 8B decoder layer on one token: the benchmark's step, decoding for one user.
        {"name": "layer_m1", "kind": "layer", "shape": "8b", "M": 1, "S": 4},
        # The same layer for sixteen sequences decoded together.
        {"name": "layer_m16", "kind": "layer", "shape": "8b", "M": 16, "S": 4},
        # The same layer on a 2048-token chunk of a prompt: the tensor-core bound end.
        {"name": "layer_m2048", "kind": "layer", "shape": "8b", "M": 2048, "S": 4},
        # A layer of somebody's own model: no dimension is a multiple of a tile, K is padded to the group length, three
        # planes, a small codebook, a bias, an odd batch.
        {"name": "linear_ragged", "kind": "linear", "M": 37, "N": 3000, "K": 3000, "S": 3, "G": 256, "form": "u8",
         "bias": True},
        # A chat turn: one user, a 512-token prompt, 64 new tokens from the 8B preset, greedy.
        {"name": "generate_b1", "kind": "generate", "shape": "8b", "layers": 32, "batch": 1, "prompt": 512, "new": 64},
        # A small server: sixteen users decoded together.
        {"name": "generate_b16", "kind": "generate", "shape": "8b", "layers": 32, "batch": 16, "prompt": 128, "new": 32},
        # Reading two long prompts of an odd length: prefill of the whole model, attention over 1500 positions.
        {"name": "prefill_2x1500", "kind": "prefill", "shape": "8b", "layers": 32, "batch": 2, "prompt": 1500},
        # Restoring a dense weight from its packed form (what loading into a dense model does per layer).
        {"name": "decode_weight", "kind": "decode", "N": 14336, "K": 4096, "S": 4, "G": 256, "form": "u16"},
        # Encoding a dense projection.
        {"name": "encode_weight", "kind": "encode", "N": 1024, "K": 4096, "S": 4},
        # Product of four encoded activation rows with an encoded weight, both sides four planes.
        {"name": "mm_t_m4", "kind": "mm_T", "M": 4, "N": 4096, "K": 4096, "LS": 4, "RS": 4},
        # A weight in the transposed encoding (groups along the outputs), the up projection of an 8B layer, one token.
        {"name": "row_deq_m1", "kind": "row_deq", "M": 1, "N": 14336, "K": 4096, "S": 4, "form": "u16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A dimension: mostly multiples of 128 as layers have them, sometimes any number."""
    v = _log(rng, lo, hi)
    return v if rng.random() < 0.35 else max(128, v // 128 * 128)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "layer", "layer", "generate", "prefill", "forward", "decode", "encode",
                       "mm_T", "row_deq"])
    if kind == "linear":
        N, K = _size(rng, 64, 32768), _size(rng, 128, 16384)
        M = min(_log(rng, 1, 4096), max(1, (1 << 36) // (N * K)))
        G = rng.choice([256, 256, 256, 128])
        return {"kind": kind, "M": M, "N": N, "K": K, "S": rng.choice([2, 3, 4, 4]), "G": G,
                "form": rng.choice(["u8", "u16", "u16", "direct"]), "bias": rng.random() < 0.3}
    if kind == "layer":
        shape = rng.choice(["tiny8", "8b", "8b", "70b"])
        return {"kind": kind, "shape": shape, "M": _log(rng, 1, 512 if shape == "70b" else 2048), "S": rng.choice([2, 3, 4, 4])}
    if kind in ("generate", "prefill", "forward"):
        shape = rng.choice(["tiny8", "8b", "8b", "70b"])
        layers = {"tiny8": 2, "8b": rng.choice([2, 4, 8]), "70b": 2}[shape]
        batch = _log(rng, 1, 16)
        prompt = min(_log(rng, 16, 2000), 4000 // batch)
        case = {"kind": kind, "shape": shape, "layers": layers, "batch": batch, "prompt": prompt}
        if kind == "generate":
            case["new"] = _log(rng, 2, 64)
        return case
    if kind == "decode":
        return {"kind": kind, "N": _size(rng, 64, 32768), "K": _size(rng, 128, 16384), "S": rng.choice([2, 3, 4, 4]),
                "G": rng.choice([256, 256, 128]), "form": rng.choice(["u8", "u16", "u16", "direct"])}
    if kind == "encode":
        return {"kind": kind, "N": _log(rng, 16, 1024), "K": _size(rng, 256, 4096), "S": rng.choice([2, 3, 4])}
    if kind == "mm_T":
        return {"kind": kind, "M": _log(rng, 1, 64), "N": _size(rng, 128, 16384), "K": 256 * _log(rng, 1, 32),
                "LS": rng.choice([2, 3, 4]), "RS": rng.choice([2, 3, 4])}
    return {"kind": kind, "M": _log(rng, 1, 32), "N": 256 * _log(rng, 1, 64), "K": _size(rng, 128, 16384),
            "S": rng.choice([2, 3, 4]), "form": rng.choice(["u8", "u16"])}


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _lines(form):
    return {"u8": 256, "u16": 4096, "direct": 0}[form]


def _packed(N, K, S, G, form, gen, scale=0.01, zero_mean=False):
    """A packed weight: even bits, coefficient lines ~ N(0, scale^2) sorted by magnitude, uniform codebook indices.
    `zero_mean`: lines that sum to zero, as those of a weight whose groups have no mean."""
    Kp = -(-K // G) * G
    bvr = torch.randint(-2 ** 31, 2 ** 31 - 1, (Kp // 32, N, S), dtype=torch.int32, device="cuda", generator=gen)
    C = _lines(form)
    lines = torch.randn((C, S) if C else (Kp // G, N, S), device="cuda", generator=gen) * scale
    if zero_mean:
        lines = lines - lines.mean(-1, keepdim=True)
    lines = torch.gather(lines, -1, lines.abs().argsort(dim=-1, descending=True)).half()
    idx = None
    if C:
        idx = torch.randint(0, C, (Kp // G, N), dtype=torch.int32, device="cuda", generator=gen)
        idx = idx.to(torch.uint8) if C <= 256 else idx.to(torch.int16).view(torch.uint16)
    return sbvr.sbvr.from_packed(bvr, idx, lines, original_shape=(N, K), group_len=G)


def _x(M, K, gen):
    return torch.randn((M, K), device="cuda", generator=gen).half()


def _config(case):
    hidden, inter, heads, kv, vocab, lines = SHAPES[case["shape"]]
    return LlamaConfig(hidden_size=hidden, intermediate_size=inter, num_hidden_layers=case["layers"],
                       num_attention_heads=heads, num_key_value_heads=kv, vocab_size=vocab, codebook_lines=lines)


def _layer_shapes(case):
    """(outputs, inputs, which activation) of q, k, v, o, gate, up, down."""
    hidden, inter, heads, kv, _, _ = SHAPES[case["shape"]]
    return [(heads * 128, hidden, 0), (kv * 128, hidden, 0), (kv * 128, hidden, 0), (hidden, heads * 128, 1),
            (inter, hidden, 2), (inter, hidden, 2), (hidden, inter, 3)]


@torch.inference_mode()
def _model(case, seed):
    """The model with the token embedding tied to the output head, permuted and raised: every token is followed clearly by one
    other, as in a trained model, so that greedy tokens do not hang on the last bit of a logit (those of random weights do)."""
    cfg = _config(case)
    ctx = case["prompt"] + case.get("new", 1)
    m = SBVRLlamaForCausalLM(cfg, device="cuda", max_batch=case["batch"], max_ctx=-(-ctx // 64) * 64).init_synthetic(seed % (1 << 31))
    head = _packed(cfg.vocab_size, cfg.hidden_size, 4, 256, "u8" if cfg.codebook_lines <= 256 else "u16", _gen(seed + 1),
                   zero_mean=True)
    m.lm_head.weight = head
    order = (torch.arange(cfg.vocab_size, device="cuda") * 10007 + 1 + seed % 1000) % cfg.vocab_size
    table = head.decode()
    raise_to = 3.0 / float(table[:1024].float().square().mean().sqrt())
    m.embed_tokens = (table * raise_to)[order]
    # one allocation for the caches of all layers: it is also what a pass returns
    caches = torch.zeros((2, cfg.num_hidden_layers) + tuple(m.kcache[0].shape), dtype=torch.float16, device="cuda")
    m.kcache, m.vcache = list(caches[0].unbind(0)), list(caches[1].unbind(0))
    return m, caches


def prepare(case, seed):
    kind, gen = case["kind"], _gen(seed)
    if kind == "linear":
        w = _packed(case["N"], case["K"], case["S"], case["G"], case["form"], gen)
        bias = torch.randn(case["N"], device="cuda", generator=gen).half() if case["bias"] else None
        return {"kind": kind, "x": _x(case["M"], case["K"], gen), "w": w, "bias": bias}
    if kind == "layer":
        shapes = _layer_shapes(case)
        form = "u8" if SHAPES[case["shape"]][5] <= 256 else "u16"
        ws = [_packed(N, K, case["S"], 256, form, gen) for N, K, _ in shapes]
        acts = {a: _x(case["M"], K, gen) for _, K, a in shapes}
        return {"kind": kind, "ws": ws, "xs": [acts[a] for _, _, a in shapes]}
    if kind in ("generate", "prefill", "forward"):
        m, caches = _model(case, seed)
        ids = torch.randint(0, m.config.vocab_size, (case["batch"], case["prompt"]), device="cuda", generator=gen)
        return {"kind": kind, "model": m, "caches": caches, "ids": ids, "new": case.get("new", 0)}
    if kind == "decode":
        return {"kind": kind, "w": _packed(case["N"], case["K"], case["S"], case["G"], case["form"], gen)}
    if kind == "encode":
        # rows of a trained projection differ in scale
        rows = torch.exp(0.25 * torch.randn((case["N"], 1), device="cuda", generator=gen))
        data = torch.randn((case["N"], case["K"]), device="cuda", generator=gen) * 0.02 * rows
        return {"kind": kind, "data": data.half(), "config": {"num_sums": case["S"]}}
    if kind == "mm_T":
        lhs = _packed(case["M"], case["K"], case["LS"], 256, "u8", gen, scale=0.5)
        return {"kind": kind, "lhs": lhs, "rhs": _packed(case["N"], case["K"], case["RS"], 256, "u16", gen)}
    # transposed: the container holds W^T, [inputs, outputs], groups of 256 along the outputs
    w_t = _packed(case["K"], case["N"], case["S"], 256, case["form"], gen)
    return {"kind": kind, "x": _x(case["M"], case["K"], gen), "w": w_t}


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return sbvr.linear(state["x"], state["w"], state["bias"])
    if kind == "layer":
        return [sbvr.linear(x, w) for x, w in zip(state["xs"], state["ws"])]
    if kind == "generate":
        return [state["model"].generate(state["ids"], state["new"]), state["caches"]]
    if kind == "prefill":
        return [state["model"].prefill(state["ids"]), state["caches"]]
    if kind == "forward":
        return [state["model"](state["ids"]), state["caches"]]
    if kind == "decode":
        return state["w"].decode()
    if kind == "encode":
        w = sbvr.sbvr(state["data"], encoder_config=state["config"], verbose_level=0)
        return [w.bvr.view(torch.int32), w.decode()]       # the codebook's length depends on the data: it comes back decoded
    if kind == "mm_T":
        return sbvr.mm_T(state["lhs"], state["rhs"])
    return sbvr.row_deq_mm_T(state["x"], state["w"])


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _weight_bytes(N, K, S, G, form):
    groups = -(-K // G)
    coeff = {"u8": groups * N + 256 * S * 2, "u16": groups * N * 2 + 4096 * S * 2, "direct": groups * N * S * 2}[form]
    return N * K * S / 8 + coeff


def work(case):
    kind = case["kind"]
    if kind == "linear":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": _weight_bytes(N, K, case["S"], case["G"], case["form"]) + 2 * (M * K + M * N), "flops": 2 * M * N * K}
    if kind == "layer":
        M, form = case["M"], "u8" if SHAPES[case["shape"]][5] <= 256 else "u16"
        shapes = _layer_shapes(case)
        return {"bytes": sum(_weight_bytes(N, K, case["S"], 256, form) + 2 * M * N for N, K, _ in shapes) +
                sum({a: 2 * M * K for _, K, a in shapes}.values()),
                "flops": sum(2 * M * N * K for N, K, _ in shapes)}
    if kind in ("generate", "prefill", "forward"):
        cfg, B, L, new = _config(case), case["batch"], case["prompt"], case.get("new", 1)
        form = "u8" if cfg.codebook_lines <= 256 else "u16"
        shapes = _layer_shapes(case)
        weights = cfg.num_hidden_layers * sum(_weight_bytes(N, K, 4, 256, form) for N, K, _ in shapes)
        head = _weight_bytes(cfg.vocab_size, cfg.hidden_size, 4, 256, form)
        kv = 2 * 2 * cfg.num_hidden_layers * cfg.num_key_value_heads * 128          # bytes of a position's keys and values
        logits = B * (L if kind == "forward" else 1)
        per_token = cfg.num_hidden_layers * sum(2 * N * K for N, K, _ in shapes)
        per_pair = cfg.num_hidden_layers * cfg.num_attention_heads * 128 * 4        # of a query and a position it attends to
        per_logits = 2 * cfg.vocab_size * cfg.hidden_size
        steps = new - 1 if kind == "generate" else 0
        return {"bytes": (weights + head) * (1 + steps) + B * L * kv + steps * B * (L + new / 2) * kv +
                (2 * logits * cfg.vocab_size if kind == "forward" else 0),
                "flops": per_token * B * (L + steps) + per_pair * B * (L * L / 2 + steps * (L + new / 2)) +
                per_logits * (logits + B * steps)}
    if kind == "decode":
        N, K = case["N"], case["K"]
        return {"bytes": _weight_bytes(N, K, case["S"], case["G"], case["form"]) + 2 * N * K, "flops": case["S"] * N * K}
    if kind == "encode":
        # every group of 256 values against one codebook of a few lines at least: a subtraction, a square and a minimum per
        # value and representable sum
        N, K, S = case["N"], case["K"], case["S"]
        return {"bytes": 2 * N * K + N * K * S / 8 + 2 * N * K / 256, "flops": 3 * N * K * 2 ** S * 10}
    if kind == "mm_T":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": _weight_bytes(M, K, case["LS"], 256, "u8") + _weight_bytes(N, K, case["RS"], 256, "u16") + 2 * M * N,
                "flops": 2 * M * N * K}
    M, N, K = case["M"], case["N"], case["K"]
    return {"bytes": _weight_bytes(K, N, case["S"], 256, case["form"]) + 2 * (M * K + M * N), "flops": 2 * M * N * K}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "encode"):
        return "exact"                             # bytes, and fp16 values with one defined rounding
    if kind in ("generate", "prefill", "forward"):
        # fp16 activations rounded some two hundred times on the way through 32 layers; a token may turn on a tie
        return {"rel": 1e-2, "differ": 0.01}
    return {"rel": 2e-3}                           # fp16 results, and weights or activations held in about 11 to 16 bits
