"""All layers of a token in one launch (mb200_decode_layers), against the oracle's restatement of the reference's layer
(src/forward.c:670-823) at the edges of that kernel's geometry."""
import numpy as np
import pytest
import torch

from oracle import oracle
from test_gpu_decode import cfg_dict, host_layer
from tests.gpu_util import layer_by_layer

pytestmark = pytest.mark.gpu

# hidden, heads, kv heads, experts, top_k, inter, V and down type, position, router
CASES = {
    "one or two rows per CTA, first position, one expert": (256, 2, 1, 3, 1, 256, 14, 0, "random"),
    "ragged rows, idle warps in the down projection": (2816, 6, 2, 17, 3, 768, 12, 15, "random"),
    "two head blocks, wide experts, ragged Q6_K down": (4096, 32, 1, 128, 8, 2816, 14, 700, "random"),
    "several tiles of positions per warp": (512, 16, 8, 8, 2, 512, 14, 5000, "random"),
    "equal logits": (1024, 4, 2, 24, 5, 512, 14, 33, "zero"),
}


@pytest.mark.parametrize("case", CASES)
def test_layers_in_one_launch_match_oracle(case):
    from mnemocuda_b200 import kernels as K
    from mnemocuda_b200.decode import DecodeConfig, ResidentModel
    K.mb200_init()
    hidden, heads, kv_heads, experts, top_k, inter, q, pos, router = CASES[case]
    cfg = DecodeConfig(n_layers=3, hidden=hidden, n_heads=heads, n_kv_heads=kv_heads, head_dim=128, n_experts=experts, top_k=top_k,
                       moe_inter=inter, vocab=512, ctx_len=pos + 1, wv_type=q, down_type=q)
    model = ResidentModel(cfg, "cuda", seed=11, kv_prefill=pos, norm_weights="random")
    if router == "zero":
        for T in model.layers:
            T["router"].zero_()
    kv = [[T[n].cpu().numpy().view(np.uint16).copy() for n in ("kv_k", "kv_v")] for T in model.layers]
    model.set_state(9, pos)
    model.step(advance=False)  # another token first: the exchange buffers hold its values
    model.set_state(5, pos)
    model.begin()
    want = model.hidden.cpu().numpy()
    for l in range(cfg.n_layers):
        want, _ = oracle.decode_layer(want, host_layer(model, l), cfg_dict(cfg), pos, kv[l][0], kv[l][1])
    model.set_state(5, pos)  # (begin() only embeds, step() does so again)
    model.step(advance=False)
    torch.cuda.synchronize()
    got = model.hidden.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - want) <= 2e-3 * np.linalg.norm(want)
    for l, T in enumerate(model.layers):  # the position's K / V rows
        for n, w in zip(("kv_k", "kv_v"), kv[l]):
            a = T[n].cpu().numpy().view(np.float16).reshape(cfg.ctx_len, -1)[pos].astype(np.float64)
            b = w.view(np.float16).reshape(cfg.ctx_len, -1)[pos].astype(np.float64)
            assert np.linalg.norm(a - b) <= 4e-3 * np.linalg.norm(b)
    assert K.mb200_device_error() == 0


def kernels_of(call):
    """How many kernels a call launches, from its capture."""
    from cuda.bindings import runtime
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    err, _, n = runtime.cudaGraphGetNodes(graph.raw_cuda_graph())
    assert int(err) == 0
    return n


def small(hidden, heads, kv_heads, experts, top_k, inter, v, down, pos, seed):
    return dict(n_layers=3, hidden=hidden, n_heads=heads, n_kv_heads=kv_heads, head_dim=128, n_experts=experts, top_k=top_k,
                moe_inter=inter, vocab=512, ctx_len=pos + 1, wv_type=v, down_type=down), pos, seed


# Both orders of sums (a one-launch expert block, kernels of its own), column groups of 1 to 8 blocks, head blocks of 16, chunk counts
EXACT = {
    "smallest": small(256, 2, 1, 3, 1, 256, 14, 14, 0, 40), "groups of one block": small(2816, 6, 2, 17, 3, 768, 12, 12, 15, 41),
    "two head blocks": small(4096, 32, 1, 128, 8, 2816, 14, 14, 700, 42), "many tiles": small(512, 16, 8, 8, 2, 512, 14, 14, 5000, 43),
    "one-launch block": small(2048, 16, 4, 16, 4, 512, 14, 12, 59, 44), "ragged groups": small(3328, 26, 2, 148, 7, 256, 12, 14, 48, 45),
    "groups of two blocks": small(2560, 24, 8, 64, 4, 2304, 14, 12, 1234, 46), "many experts": small(1024, 8, 8, 148, 8, 1024, 14, 14, 6, 47),
    "wide": small(4096, 64, 4, 100, 5, 768, 14, 14, 2047, 48),
    # whole models: a rounding more or less ends, by way of a router, in another token at some of these
    "30B, position 4095, seed 1": ("qwen3_30b", 4095, 1), "30B, position 4095, seed 4": ("qwen3_30b", 4095, 4),
    "30B, position 2000, seed 21": ("qwen3_30b", 2000, 21), "30B, position 776, seed 3": ("qwen3_30b", 776, 3),
    "235B, position 8191, seed 2": ("qwen3_235b", 8191, 2), "235B, position 103, seed 4": ("qwen3_235b", 103, 4),
}


@pytest.mark.parametrize("case", EXACT)
def test_one_launch_is_layer_by_layer_to_the_bit(case):
    """The hidden vector after every layer, the K / V rows, logits and token. Deep synthetic models magnify a rounding until a router
    picks another expert, so no tolerance would tell an error from a rounding."""
    from mnemocuda_b200 import kernels as K
    from mnemocuda_b200.decode import DecodeConfig, ResidentModel
    K.mb200_init()
    shape, pos, seed = EXACT[case]
    whole = isinstance(shape, str)
    cfg = DecodeConfig(**shape) if not whole else getattr(DecodeConfig, shape)(n_layers=48 if shape == "qwen3_30b" else 8)
    model = ResidentModel(cfg, "cuda", seed=seed, kv_prefill=pos, norm_weights="ones" if whole else "random")
    rows = lambda: [T[n][pos].clone() for T in model.layers for n in ("kv_k", "kv_v")]
    model.set_state(seed, pos)
    model.begin()
    want = []
    for l in range(cfg.n_layers):
        layer_by_layer(model, l)
        want.append(model.hidden.clone())
    model.finish(advance=False)
    want_rows, want_logits, want_token = rows(), model.logits.clone(), int(model.token.item())
    for T in model.layers:
        T["kv_k"][pos], T["kv_v"][pos] = 0, 0
    model.set_state(seed, pos)
    model.begin()
    assert kernels_of(lambda: model.layer(0)) == 1
    for l in range(cfg.n_layers):
        model.layer(l)
        assert torch.equal(model.hidden, want[l]), l
    assert all(torch.equal(a, b) for a, b in zip(rows(), want_rows))
    for T in model.layers:
        T["kv_k"][pos], T["kv_v"][pos] = 0, 0
    model.set_state(seed, pos)
    model.step(advance=False)
    assert torch.equal(model.hidden, want[-1]) and torch.equal(model.logits, want_logits) and int(model.token.item()) == want_token
    assert all(torch.equal(a, b) for a, b in zip(rows(), want_rows))
    assert K.mb200_device_error() == 0


@pytest.mark.parametrize("pos", [0, 5, 16, 23, 30, 47])
def test_unwritten_cache_rows_do_not_matter(pos):
    """The cache holds NaN from the position on, where nothing has been stored yet, in both forms of a layer (32 query heads on a KV
    head: two blocks of them read the row that one stores)."""
    from mnemocuda_b200 import kernels as K
    from mnemocuda_b200.decode import DecodeConfig, ResidentModel
    K.mb200_init()
    cfg = DecodeConfig(n_layers=2, hidden=2048, n_heads=32, n_kv_heads=1, head_dim=128, n_experts=16, top_k=4, moe_inter=512, vocab=512,
                       ctx_len=64)
    model = ResidentModel(cfg, "cuda", seed=3, kv_prefill=pos, norm_weights="random")
    got = {}
    for fill in (0.0, float("nan")):
        for form in (model.layer, lambda l: layer_by_layer(model, l)):
            for T in model.layers:
                T["kv_k"][pos:], T["kv_v"][pos:] = fill, fill
            model.set_state(9, pos)
            model.begin()
            for l in range(cfg.n_layers):
                form(l)
            got[fill, form] = model.hidden.clone()
            assert torch.isfinite(model.hidden).all()
    want = list(got.values())[0]
    assert all(torch.equal(h, want) for h in got.values())
