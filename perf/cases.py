"""What is timed of this library, and on which inputs: the work its users have it do, through its public calls.

The path has two directions. Decode (batch 1): quantised matvecs, the routed expert block, attention over the KV cache,
whole tokens, sampling. Prefill (a batch of tokens): the tensor-core GEMM and its grouped per-expert form. Shapes are
those of this repository's configurations (the 30B-A3B and 235B-A22B shapes of mnemocuda_b200/decode.py and moe.py)
and odd sizes around them. Weights are synthetic GGUF blocks with the distributions of mnemocuda_b200/synth.py.

A case is a dict with a "kind"; listed() has the cases that are always timed, draw() gives more of the same ranges.
Launches use programmatic dependent launch, as a serving program's would (weights are written once, at load).
"""
from __future__ import annotations

import math

import torch

from mnemocuda_b200 import kernels as K
from mnemocuda_b200 import synth
from mnemocuda_b200.decode import DecodeConfig, ResidentModel
from mnemocuda_b200.moe import HostMoEBlock, MoEShape, ResidentMoE

# weight type -> (columns per block, bytes per block, public call)
TYPES = {
    "q4k": (256, synth.Q4K_BLOCK, K.cuda_matvec_q4k),
    "q6k": (256, synth.Q6K_BLOCK, K.cuda_matvec_q6k),
    "q8_0": (32, synth.Q8_0_BLOCK, K.cuda_matvec_q8_0),
    "q5k": (256, synth.Q5K_BLOCK, K.cuda_matvec_q5k),
    "q3k": (256, synth.Q3K_BLOCK, K.cuda_matvec_q3k),
}
# byte offsets of a block's fp16 scales and their spread (the other bytes are uniform)
SCALES = {"q8_0": ((0,), 2e-3), "q5k": ((0, 2), 2e-3), "q3k": ((108,), 2e-3)}
# expert blocks of the two configured model shapes; others are drawn around them
EXPERTS_235B = {"H": 4096, "eff": 1536, "experts": 128, "top_k": 8}
EXPERTS_30B = {"H": 2048, "eff": 768, "experts": 128, "top_k": 8}


def listed():
    return [
        # the K projection of one 30B-shape layer, one call: the smallest, all latency
        {"name": "matvec_q4k_512x2048", "kind": "matvec", "type": "q4k", "rows": 512, "cols": 2048, "layers": 1, "graph": False},
        # one projection of the 235B shape through sixteen layers, captured once and replayed: the ordinary decode matvec
        {"name": "matvec_q4k_8192x4096_16_layers", "kind": "matvec", "type": "q4k", "rows": 8192, "cols": 4096, "layers": 16, "graph": True},
        # another weight type, rows and blocks per row that divide by nothing
        {"name": "matvec_q5k_5461x2816", "kind": "matvec", "type": "q5k", "rows": 5461, "cols": 2816, "layers": 1, "graph": False},
        # the expert block of four layers of the 235B shape (router, top-8, gate/up, down) inside a captured decode
        {"name": "moe_block_235b_4_layers", "kind": "moe_block", **EXPERTS_235B, "layers": 4},
        # the same block for an engine that keeps the hidden state in host memory, one call per layer
        {"name": "moe_block_host_235b", "kind": "moe_block_host", **EXPERTS_235B, "layers": 1},
        # whole tokens: the complete 30B shape at the end of its context, and a slice of the 235B shape's layers
        {"name": "decode_30b_ctx4096", "kind": "decode", "shape": "30b", "layers": 48, "pos": 4095},
        {"name": "decode_235b_8_layers_ctx8192", "kind": "decode", "shape": "235b", "layers": 8, "pos": 8191},
        # prefill: the dense GEMM of a 512-token chunk, a short odd prompt on the other weight type, the expert block of a chunk
        {"name": "gemm_q4k_512x8192x4096", "kind": "gemm", "type": "q4k", "M": 512, "N": 8192, "K": 4096},
        {"name": "gemm_q6k_197x4096x1536", "kind": "gemm", "type": "q6k", "M": 197, "N": 4096, "K": 1536},
        {"name": "moe_prefill_235b_512", "kind": "moe_prefill", **EXPERTS_235B, "M": 512},
        # the INT8 KV cache at a long context
        {"name": "attention_int8_64x4_ctx32768", "kind": "attention", "cache": "int8", "heads": 64, "kv_heads": 4, "seq": 32768},
        # temperature / top-p sampling over the vocabulary
        {"name": "sample_top_p_151936", "kind": "sample", "vocab": 151936, "temperature": 0.7, "top_p": 0.9},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_experts(rng):
    if rng.random() < 0.5:
        return dict(rng.choice([EXPERTS_235B, EXPERTS_30B]))
    return {"H": 256 * rng.choice([4, 6, 8, 10, 11, 12, 16]), "eff": 256 * _log_int(rng, 1, 6), "experts": rng.choice([16, 60, 64, 128]),
            "top_k": rng.choice([4, 6, 8])}


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "gemm", "gemm", "moe_prefill", "moe_block", "moe_block_host", "decode", "attention", "sample"])
    if kind == "matvec":
        # from a KV projection to a vocabulary; a row of the widest tensors is a feed-forward width
        t = rng.choice(["q4k", "q4k", "q6k", "q6k", "q8_0", "q5k", "q3k"])
        rows, cols = _log_int(rng, 256, 151936), 256 * _log_int(rng, 4, 48)
        rows = min(rows, 151936 * 4096 // cols)
        layers = rng.choice([1, 1, 4, 16]) if rows * cols <= 8192 * 4096 else 1
        return {"kind": kind, "type": t, "rows": rows, "cols": cols, "layers": layers, "graph": layers > 1}
    if kind == "gemm":
        return {"kind": kind, "type": rng.choice(["q4k", "q6k"]), "M": _log_int(rng, 8, 2048), "N": _log_int(rng, 512, 8192),
                "K": 256 * _log_int(rng, 4, 32)}
    if kind == "moe_prefill":
        e = _draw_experts(rng)
        return {"kind": kind, **e, "M": _log_int(rng, 16, 512 * 4096 * 1536 / (e["H"] * e["eff"]))}
    if kind in ("moe_block", "moe_block_host"):
        return {"kind": kind, **_draw_experts(rng), "layers": rng.randint(1, 6)}
    if kind == "decode":
        shape = rng.choice(["235b", "30b"])
        return {"kind": kind, "shape": shape, "layers": rng.randint(2, 8) if shape == "235b" else rng.randint(4, 16),
                "pos": _log_int(rng, 32, 8191 if shape == "235b" else 4095)}
    if kind == "attention":
        heads, kv = rng.choice([(32, 4), (64, 4), (32, 8), (64, 8)])
        return {"kind": kind, "cache": rng.choice(["f16", "int8"]), "heads": heads, "kv_heads": kv, "seq": _log_int(rng, 64, 32768)}
    return {"kind": kind, "vocab": _log_int(rng, 32000, 151936), "temperature": round(rng.uniform(0.4, 1.2), 2),
            "top_p": round(rng.uniform(0.7, 1.0), 2)}


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _weights(type_, n_blocks, seed, g):
    """n_blocks blocks of one type as device bytes."""
    bb = TYPES[type_][1]
    w = torch.empty(n_blocks * bb, dtype=torch.uint8, device="cuda")
    if type_ == "q4k":
        K.mb200_fill_q4k(w, n_blocks, seed)
    elif type_ == "q6k":
        K.mb200_fill_q6k(w, n_blocks, seed)
    else:
        w.random_(0, 256, generator=g)
        offsets, spread = SCALES[type_]
        for o in offsets:
            d = (torch.randn(n_blocks, device="cuda", generator=g).abs() * spread).half()
            w.view(n_blocks, bb)[:, o:o + 2] = d.view(torch.uint8).view(n_blocks, 2)
    return w


def _captured(call):
    """`call` as a CUDA graph, after one eager pass."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    return graph


def _config(case):
    if case["shape"] == "30b":
        return DecodeConfig.qwen3_30b(n_layers=case["layers"])
    return DecodeConfig.qwen3_235b(n_layers=case["layers"])


def _expert_shape(case):
    return MoEShape(case["experts"], case["top_k"], case["H"], case["eff"])


def prepare(case, seed):
    K.mb200_init()
    K.mb200_set_pdl(True)
    g = torch.Generator(device="cuda").manual_seed(seed)
    randn = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    kind = case["kind"]
    s = {"case": case}
    if kind == "matvec":
        per, bb, call = TYPES[case["type"]]
        rows, cols, layers = case["rows"], case["cols"], case["layers"]
        nb = rows * (cols // per)
        s["w"] = [_weights(case["type"], nb, seed * 64 + l, g) for l in range(layers)]
        s["x"] = [randn(cols) for _ in range(layers)]
        s["y"] = [torch.empty(rows, device="cuda") for _ in range(layers)]
        s["call"] = call
        if case["graph"]:
            s["graph"] = _captured(lambda: [call(w, x, y, rows, cols) for w, x, y in zip(s["w"], s["x"], s["y"])])
    elif kind in ("moe_block", "moe_block_host"):
        H, layers = case["H"], case["layers"]
        moe = s["moe"] = ResidentMoE(_expert_shape(case), layers, seed=seed)
        s["x"], s["residual"] = randn(layers, H), randn(layers, H)
        s["out"] = torch.empty(layers, H, device="cuda")
        if kind == "moe_block":
            s["graph"] = _captured(lambda: [moe.forward(l, s["x"][l], s["residual"][l], s["out"][l]) for l in range(layers)])
        else:
            s["block"] = HostMoEBlock(moe)
            s["x_res"] = torch.stack([s["x"], s["residual"]], dim=1).cpu().pin_memory()
            s["host_out"] = torch.empty(layers, H).pin_memory()
    elif kind == "decode":
        # the cache holds the positions before `pos`; one pass decodes the token at `pos` (and stays there)
        m = s["model"] = ResidentModel(_config(case), seed=seed, kv_prefill=case["pos"])
        m.set_state(seed % m.cfg.vocab, case["pos"])
        s["graph"] = m.capture(1, advance=False)
    elif kind == "gemm":
        s["w"] = _weights(case["type"], case["N"] * (case["K"] // 256), seed, g)
        s["x"] = randn(case["M"], case["K"]).half()
        s["y"] = torch.empty(case["M"], case["N"], device="cuda")
        s["call"] = K.mb200_gemm_q4k_f16 if case["type"] == "q4k" else K.mb200_gemm_q6k_f16
    elif kind == "moe_prefill":
        H, M = case["H"], case["M"]
        moe = s["moe"] = ResidentMoE(_expert_shape(case), 1, seed=seed)
        s["x"], s["residual"] = randn(M, H).half(), randn(M, H)
        # routing as the router gives it, with some experts in more demand than others
        logits = s["x"].float() @ moe.router[0].T + 0.5 * randn(case["experts"])
        top = torch.topk(logits, case["top_k"], dim=1)
        s["ids"], s["wts"] = top.indices.int().contiguous(), torch.softmax(top.values, dim=1).contiguous()
        n = K.mb200_moe_prefill_workspace_bytes(M, case["top_k"], H, case["eff"], case["experts"]) + 256
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        s["ws"] = ws[-ws.data_ptr() % 256:]
        s["y"] = torch.empty(M, H, device="cuda")
    elif kind == "attention":
        heads, kv, seq = case["heads"], case["kv_heads"], case["seq"]
        s["q"], s["out"] = randn(heads, 128), torch.empty(heads, 128, device="cuda")
        k, v = randn(seq, kv, 128), randn(seq, kv, 128)
        if case["cache"] == "f16":
            s["k"], s["v"] = k.half(), v.half()
        else:
            ks, vs = k.abs().amax(-1) / 127, v.abs().amax(-1) / 127
            s["k"], s["v"] = (k / ks[..., None]).round().to(torch.int8), (v / vs[..., None]).round().to(torch.int8)
            s["ks"], s["vs"] = ks.contiguous(), vs.contiguous()
    elif kind == "sample":
        s["logits"] = 3 * randn(case["vocab"])
        s["rng"] = (seed * 0x9E3779B97F4A7C15 + 1) & (2 ** 64 - 1)
        s["token"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    else:
        raise ValueError(kind)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "matvec":
        if case["graph"]:
            s["graph"].replay()
        else:
            s["call"](s["w"][0], s["x"][0], s["y"][0], case["rows"], case["cols"])
        return s["y"]
    if kind == "moe_block":
        s["graph"].replay()
        return s["out"], s["moe"].ids, s["moe"].wts
    if kind == "moe_block_host":
        for l in range(case["layers"]):
            s["block"](l, s["x_res"][l], s["host_out"][l])
        return s["host_out"], s["moe"].ids, s["moe"].wts
    if kind == "decode":
        m = s["model"]
        s["graph"].replay()
        return m.token, m.logits, m.hidden, m.layers[-1]["kv_k"], m.layers[-1]["kv_v"]
    if kind == "gemm":
        s["call"](s["w"], s["x"], s["y"], case["M"], case["N"], case["K"])
        return s["y"]
    if kind == "moe_prefill":
        m = s["moe"].shape
        K.mb200_moe_prefill(s["moe"].experts[0], m.stride, m.gate_sz, m.up_sz, m.down_type, m.NE, m.K, m.H, m.EFF, s["x"],
                            s["ids"], s["wts"], s["residual"], s["y"], case["M"], 0, s["ws"])
        return s["y"]
    if kind == "attention":
        heads, kv, seq = case["heads"], case["kv_heads"], case["seq"]
        if case["cache"] == "f16":
            K.cuda_attention_f16kv(s["q"], s["k"], s["v"], s["out"], heads, 128, kv, seq, heads // kv, 128 ** -0.5)
        else:
            K.cuda_attention_int8kv(s["q"], s["k"], s["v"], s["ks"], s["vs"], s["out"], heads, 128, kv, seq, heads // kv, 128 ** -0.5)
        return s["out"]
    K.cuda_sample_token(s["logits"], case["vocab"], case["temperature"], case["top_p"], s["rng"], s["token"])
    return s["token"]


# ---- what a pass cannot do without, and how close another correct implementation comes ------------------------------

def work(case):
    kind = case["kind"]
    if kind == "matvec":
        per, bb, _ = TYPES[case["type"]]
        rows, cols, n = case["rows"], case["cols"], case["layers"]
        return {"bytes": n * (rows * (cols // per) * bb + 4 * (rows + cols)), "flops": 2 * n * rows * cols}
    if kind in ("moe_block", "moe_block_host"):
        m, n = _expert_shape(case), case["layers"]
        return {"bytes": n * (m.algorithmic_bytes + 12 * m.H), "flops": 2 * n * (m.NE * m.H + m.K * 3 * m.H * m.EFF)}
    if kind == "decode":
        c = _config(case)
        seq = case["pos"] + 1
        per_layer = 2 * c.hidden * c.q_dim + 2 * c.hidden * c.kv_dim + c.n_experts * c.hidden + c.top_k * 3 * c.hidden * c.moe_inter
        return {"bytes": c.algorithmic_bytes_per_token(seq) + 4 * c.vocab,
                "flops": 2 * (c.n_layers * (per_layer + 2 * seq * c.q_dim) + c.vocab * c.hidden)}
    if kind == "gemm":
        M, N, Kd = case["M"], case["N"], case["K"]
        return {"bytes": N * (Kd // 256) * TYPES[case["type"]][1] + 2 * M * Kd + 4 * M * N, "flops": 2 * M * N * Kd}
    if kind == "moe_prefill":
        m, M = _expert_shape(case), case["M"]
        used = m.NE * (1 - (1 - m.K / m.NE) ** M)  # experts that any token reaches, evenly routed
        return {"bytes": used * m.stride + M * (2 * m.H + 4 * m.H + 4 * m.H + 8 * m.K), "flops": 2 * M * m.K * 3 * m.H * m.EFF}
    if kind == "attention":
        seq, kv, heads = case["seq"], case["kv_heads"], case["heads"]
        per = 2 * 128 if case["cache"] == "f16" else 128 + 4
        return {"bytes": 2 * seq * kv * per + 8 * heads * 128, "flops": 4 * seq * heads * 128}
    return {"bytes": 4 * case["vocab"] + 4, "flops": 4 * case["vocab"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "matvec":
        return {"rel": 5e-5, "max": 1e-3}   # activations carry two int8 levels (1e-5), sums are fp32
    if kind in ("moe_block", "moe_block_host"):
        return {"rel": 2e-4, "max": 4e-3}   # two such products in a row around SwiGLU
    if kind == "decode":
        return {"rel": 2e-3, "max": 5e-2}   # tens of layers of them, and an fp16 cache
    if kind == "gemm":
        return {"rel": 6e-4, "max": 1e-2}   # weights rounded to fp16 for the tensor cores
    if kind == "moe_prefill":
        return {"rel": 5e-4, "max": 2e-2}   # two GEMMs in a row on split fp16 operands
    if kind == "attention":
        # fp16 cache: probabilities in fp16; int8 cache: fp32 arithmetic on exact integers
        return {"rel": 5e-4, "max": 1e-2} if case["cache"] == "f16" else {"rel": 5e-5, "max": 1e-3}
    return "exact"
