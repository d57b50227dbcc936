"""All layers of a token in one launch (mb200_decode_layers), against the oracle's restatement of the reference's layer
(src/forward.c:670-823) at the edges of that kernel's geometry."""
import numpy as np
import pytest
import torch

from oracle import oracle
from test_gpu_decode import cfg_dict, host_layer

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
