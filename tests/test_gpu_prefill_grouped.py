"""Grouped prefill at the edges of its tiles: token counts around 16 / 32 / 64 / 128 per expert (the box classes and the
accumulator split), one super-block per row, an odd number of them, Q4_K and Q6_K down, sixteen slots; against the oracle's
per-token expert sequence."""
import numpy as np
import pytest
import torch

from mnemocuda_b200 import synth
from oracle import oracle
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from mnemocuda_b200 import kernels
    kernels.mb200_init()
    return kernels


@pytest.mark.parametrize("counts,H,EFF,down", [((1, 15, 16, 17, 31, 32, 33), 256, 256, 14), ((63, 64, 65, 3), 768, 256, 14),
                                               ((127, 128, 129, 0, 40), 256, 768, 14), ((260, 5, 33), 512, 256, 12)])
def test_token_counts_at_tile_edges(K, counts, H, EFF, down):
    NE, M = len(counts), sum(counts)
    g, u, d = synth.expert_sizes(H, EFF, down)
    stride = g + u + d
    experts = np.concatenate([synth.expert_blob(1800 + e, H, EFF, down) for e in range(NE)])
    x = synth.normal_f16(1801, M * H).reshape(M, H)
    ids = np.random.default_rng(1802).permutation(np.repeat(np.arange(NE), counts)).astype(np.int32).reshape(M, 1)
    wts = (0.5 + np.random.default_rng(1803).random((M, 1))).astype(np.float32)
    n = K.mb200_moe_prefill_workspace_bytes(M, 1, H, EFF, NE)
    ws = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
    ws = ws[-ws.data_ptr() % 256:]
    y = torch.full((M, H), float("nan"), device="cuda")
    K.mb200_moe_prefill(dev(experts), stride, g, u, down, NE, 1, H, EFF, dev(x), dev(ids), dev(wts), None, y, M, 0, ws)
    got = host(y).astype(np.float64)
    for t in range(M):
        e = int(ids[t, 0])
        want = oracle.expert_fwd(experts[e * stride:(e + 1) * stride], g, u, H, EFF, down, float(wts[t, 0]), x[t].astype(np.float32),
                                 np.zeros(H, np.float32)).astype(np.float64)
        assert np.linalg.norm(got[t] - want) <= 3e-4 * np.linalg.norm(want), (t, e)
    assert K.mb200_device_error() == 0
