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


@pytest.mark.parametrize("d,scale,dmin,m", [(0.0005245209, 19, 0.0014314651, 63), (0.0025806427, 1, 0.004219055, 5),
                                            (0.00076055527, 57, 0.0061187744, 50)])
def test_q4k_scales_that_round_up_to_the_next_power_of_two(K, d, scale, dmin, m):
    """16 s + b of these sub-blocks lies just below a power of two and, rounded to the unit of the exact half of the split, just above it.
    Gate and up of such sub-blocks only, against fp64; the bound is twelve times what fp32 accumulation over K leaves (1e-5) and a tenth
    of what a weight off by one unit everywhere would (1e-3)."""
    H, EFF, M = 512, 256, 24
    rng = np.random.default_rng(6)
    blocks = rng.integers(0, 256, (2 * EFF * H // 256, synth.Q4K_BLOCK)).astype(np.uint8)
    blocks[:, :4] = np.array([d, dmin], np.float16).view(np.uint8)
    blocks[:, 4:8] = scale | (scale >> 4 << 6)
    blocks[:, 8:12] = m | (m >> 4 << 6)
    blocks[:, 12:16] = (scale & 15) | ((m & 15) << 4)
    g, u, dn = synth.expert_sizes(H, EFF, 14)
    expert = np.concatenate([blocks.reshape(-1), synth.q6k_matrix(7, H, EFF).reshape(-1)])
    x = rng.standard_normal((M, H)).astype(np.float16)
    n = K.mb200_moe_prefill_workspace_bytes(M, 1, H, EFF, 1)
    ws = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
    ws = ws[-ws.data_ptr() % 256:]
    y = torch.empty(M, H, device="cuda")
    K.mb200_moe_prefill(dev(expert), g + u + dn, g, u, 14, 1, 1, H, EFF, dev(x), dev(np.zeros((M, 1), np.int32)),
                        dev(np.ones((M, 1), np.float32)), None, y, M, 0, ws)
    w = oracle.dequant_q4k(blocks.reshape(-1), 2 * EFF, H).astype(np.float64)
    gate, up = x.astype(np.float64) @ w[:EFF].T, x.astype(np.float64) @ w[EFF:].T
    want = (gate / (1 + np.exp(-gate)) * up) @ oracle.dequant_q6k(expert[g + u:], H, EFF).astype(np.float64).T
    err = np.linalg.norm(host(y) - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() <= 1.2e-4, err.max()
    assert K.mb200_device_error() == 0


def test_q6k_weights_keep_22_bits(K):
    """One column of each expert's down projection at a time: a token's input picks it by way of a gate / up row of its own. Each
    result is a weight times a known activation, off by the weight's two halves (4.4e-7), the activation's (2.4e-7) and fp32 rounding."""
    H, EFF, NE = 256, 256, 6
    g, u, d = synth.expert_sizes(H, EFF, 14)
    rng = np.random.default_rng(8)
    experts, want = [], []
    for e in range(NE):
        gate_up = np.zeros((2 * EFF, H // 256, synth.Q4K_BLOCK), np.uint8)
        col = int(rng.integers(0, EFF))
        for row in (col, EFF + col):  # 3 / 16 in column 0, nothing elsewhere
            gate_up[row, 0, :2] = np.array([1 / 16], np.float16).view(np.uint8)
            gate_up[row, 0, 4] = 1
            gate_up[row, 0, 16] = 3
        down = synth.q6k_matrix(900 + e, H, EFF).reshape(H, -1)
        down[:, 192:208] = rng.integers(0, 256, (H, 16))  # scales of all eight bits
        experts.append(np.concatenate([gate_up.reshape(-1), down.reshape(-1)]))
        a = 3.0 * 3.0 / (1 + np.exp(-3.0))
        want.append(a * oracle.dequant_q6k(down.reshape(-1), H, EFF).astype(np.float64)[:, col])
    x = np.zeros((NE, H), np.float16)
    x[:, 0] = 16
    n = K.mb200_moe_prefill_workspace_bytes(NE, 1, H, EFF, NE)
    ws = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
    ws = ws[-ws.data_ptr() % 256:]
    y = torch.empty(NE, H, device="cuda")
    K.mb200_moe_prefill(dev(np.concatenate(experts)), g + u + d, g, u, 14, NE, 1, H, EFF, dev(x), dev(np.arange(NE, dtype=np.int32).reshape(NE, 1)),
                        dev(np.ones((NE, 1), np.float32)), None, y, NE, 0, ws)
    got, want = host(y).astype(np.float64), np.array(want)
    assert np.all(np.abs(got - want) <= 1e-6 * np.abs(want))
    assert K.mb200_device_error() == 0


@pytest.mark.parametrize("counts,H,EFF,down", [((5, 33), 1280, 512, 14), ((40, 0, 64), 256, 1024, 14), ((65, 32), 512, 2048, 14),
                                               ((1, 96), 2304, 1280, 12), ((31, 66), 256, 256, 12)])
def test_rows_per_group_and_sums_of_activations(K, counts, H, EFF, down):
    """Q6_K down rows taken 8, 4, 2 and 1 at a time (EFF / 256 odd, 2, 4, 8), activation sums of one, one over four and nine super-blocks
    a row, both accumulators of a tile full, nearly empty and unused; against fp64. Weights are exact here and activations pairs of
    halves (2^-22), so what is left is fp32 accumulation, 1.5e-6; weights rounded to fp16 once would be off by 2.4e-4."""
    NE, M = len(counts), sum(counts)
    g, u, d = synth.expert_sizes(H, EFF, down)
    experts = [synth.expert_blob(1900 + e, H, EFF, down) for e in range(NE)]
    x = synth.normal_f16(1901, M * H).reshape(M, H)
    ids = np.random.default_rng(1902).permutation(np.repeat(np.arange(NE), counts)).astype(np.int32).reshape(M, 1)
    n = K.mb200_moe_prefill_workspace_bytes(M, 1, H, EFF, NE)
    ws = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
    ws = ws[-ws.data_ptr() % 256:]
    y = torch.full((M, H), float("nan"), device="cuda")
    K.mb200_moe_prefill(dev(np.concatenate(experts)), g + u + d, g, u, down, NE, 1, H, EFF, dev(x), dev(ids), dev(np.ones((M, 1), np.float32)), None,
                        y, M, 0, ws)
    got = host(y).astype(np.float64)
    for e in range(NE):
        t = ids[:, 0] == e
        w = oracle.dequant_q4k(experts[e][:g + u], 2 * EFF, H).astype(np.float64)
        w2 = (oracle.dequant_q6k if down == 14 else oracle.dequant_q4k)(experts[e][g + u:g + u + d], H, EFF).astype(np.float64)
        gate, up = x[t].astype(np.float64) @ w[:EFF].T, x[t].astype(np.float64) @ w[EFF:].T
        want = (gate / (1 + np.exp(-gate)) * up) @ w2.T
        assert np.all(np.linalg.norm(got[t] - want, axis=1) <= 2e-5 * np.linalg.norm(want, axis=1)), e
    assert K.mb200_device_error() == 0


def test_swiglu_between_the_gemms_rounds_as_fp32_does(K):
    """gate / (1 + exp(-gate)) to one rounding of the sum and one of the quotient: 2^-23 of the value, plus 2^-27 for an exponential off by two
    units (gate >= 4). Row i of gate and up picks x[i] and x[255], rows of the down projection are unit vectors, scaling is by powers of two,
    and values whose pair of halves would round once more are left out."""
    H, EFF, M = 256, 256, 64
    g, u, d = synth.expert_sizes(H, EFF, 14)
    gate_up = np.zeros((2 * EFF, synth.Q4K_BLOCK), np.uint8)
    for row in range(EFF):
        for r, col in ((row, row), (EFF + row, 255)):
            sub = col // 32
            gate_up[r, :2] = np.array([1.0], np.float16).view(np.uint8)
            gate_up[r, 4 + sub if sub < 4 else 8 + sub] = 1  # scale 1 of this sub-block
            gate_up[r, 16 + 32 * (sub // 2) + col % 32] = 1 << 4 * (sub & 1)
    assert np.array_equal(oracle.dequant_q4k(gate_up[:EFF].reshape(-1), EFF, H), np.eye(EFF, dtype=np.float32))
    down = np.zeros((H, synth.Q6K_BLOCK), np.uint8)
    down[:, 128:192] = 0xAA  # q - 32 = 0: low nibbles 0, high bits 2
    down[:, 192:208] = 1
    down[:, 208:] = np.array([1.0], np.float16).view(np.uint8)
    for row in range(H):  # q - 32 = 1 in column `row`
        half, i = row // 128, row % 128
        down[row, 64 * half + i % 64] |= 1 << 4 * (i // 64)
    assert np.array_equal(oracle.dequant_q6k(down.reshape(-1), H, EFF), np.eye(H, dtype=np.float32))
    expert = np.concatenate([gate_up.reshape(-1), down.reshape(-1)])
    x = np.random.default_rng(9).uniform(4, 15, (M, H)).astype(np.float16)
    x[:, 255] = 16
    n = K.mb200_moe_prefill_workspace_bytes(M, 1, H, EFF, 1)
    ws = torch.empty(n + 256, dtype=torch.uint8, device="cuda")
    ws = ws[-ws.data_ptr() % 256:]
    y = torch.empty(M, H, device="cuda")
    K.mb200_moe_prefill(dev(expert), g + u + d, g, u, 14, 1, 1, H, EFF, dev(x), dev(np.zeros((M, 1), np.int32)),
                        dev(np.ones((M, 1), np.float32)), None, y, M, 0, ws)
    gate = x.astype(np.float64)
    want = gate / (1 + np.exp(-gate))  # times 16 of up, times 1 / 16 on the way through the halves, which the result has back
    unit = 2.0 ** np.floor(np.log2(want))
    exact = np.abs(want - want.astype(np.float16)) < 0.99 * 2.0 ** -12 * unit  # what the low half holds has 11 bits
    err = np.abs(host(y).astype(np.float64) / 16 - want) / want
    assert exact.sum() > 4000 and err[exact].max() <= 2.0 ** -23 + 2.0 ** -27, (err[exact].max(), exact.sum())
    assert K.mb200_device_error() == 0
