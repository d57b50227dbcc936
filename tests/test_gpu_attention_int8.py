"""The tensor-core attention over the INT8 cache at the edges of its tiles, chunks and head blocks, and the sampler
beyond the vocabulary size whose candidates all fit one list per thread (both against the C oracle)."""
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


# one chunk / one cluster / several clusters; a position past a tile and past a chunk; 1, 3, 16 and 20 heads per KV head
@pytest.mark.parametrize("nh,nkv,S", [(4, 4, 16), (16, 1, 17), (64, 4, 128), (64, 4, 129), (12, 4, 255), (20, 1, 1025),
                                      (40, 2, 2049), (32, 8, 4097)])
@pytest.mark.parametrize("spread", [1.0, 1e6])
def test_int8_attention_edges(K, nh, nkv, S, spread):
    """spread: V scales that differ by that factor from position to position (they are folded into fp16 operands)."""
    rng = np.random.default_rng(S + nh)
    k8 = rng.integers(-127, 128, (S, nkv, 128), dtype=np.int8)
    v8 = rng.integers(-127, 128, (S, nkv, 128), dtype=np.int8)
    ks = ((0.5 + rng.random((S, nkv))) / 127).astype(np.float32)
    vs = (spread ** -rng.random((S, nkv)) / 127).astype(np.float32)
    q = synth.normal_f32(4100 + S, nh * 128)
    want = oracle.attention_int8kv(q, k8, v8, ks, vs, nh, 128, nkv, S, nh // nkv, 128 ** -0.5).reshape(nh, 128).astype(np.float64)
    out = torch.full((nh * 128,), float("nan"), device="cuda")
    for _ in range(2):  # twice: the tickets must be back at zero
        out.fill_(float("nan"))
        K.cuda_attention_int8kv(dev(q), dev(k8), dev(v8), dev(ks), dev(vs), out, nh, 128, nkv, S, nh // nkv, 128 ** -0.5)
        got = host(out).reshape(nh, 128).astype(np.float64)
        rel = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert rel.max() <= 2e-5, rel.max()


@pytest.mark.parametrize("nh,nkv,S", [(4, 4, 33), (16, 2, 129), (40, 2, 300)])
def test_int8_attention_query_range(K, nh, nkv, S):
    """Heads whose q lies ten decades apart, with scores of order one by way of the K scales: q itself does not fit fp16."""
    rng = np.random.default_rng(S)
    k8 = rng.integers(-127, 128, (S, nkv, 128), dtype=np.int8)
    v8 = rng.integers(-127, 128, (S, nkv, 128), dtype=np.int8)
    vs = ((0.5 + rng.random((S, nkv))) / 127).astype(np.float32)
    for size in (1e-9, 1.0, 1e7, 1e12):
        ks = ((0.5 + rng.random((S, nkv))) / 127 / size).astype(np.float32)
        q = synth.normal_f32(4200 + S, nh * 128).reshape(nh, 128) * np.float32(size)
        q[1::3] *= np.float32(1e-5)
        want = oracle.attention_int8kv(q.reshape(-1), k8, v8, ks, vs, nh, 128, nkv, S, nh // nkv, 128 ** -0.5).reshape(nh, 128).astype(np.float64)
        out = torch.empty(nh * 128, device="cuda")
        K.cuda_attention_int8kv(dev(q.reshape(-1)), dev(k8), dev(v8), dev(ks), dev(vs), out, nh, 128, nkv, S, nh // nkv, 128 ** -0.5)
        got = host(out).reshape(nh, 128).astype(np.float64)
        rel = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert rel.max() <= 2e-5, (size, rel.max())


@pytest.mark.parametrize("gqa", [1, 8, 9, 16])
@pytest.mark.parametrize("ramp", [1, -1, 0])
def test_int8_attention_moving_maxima(K, gqa, ramp):
    """Scores and V scales that rise, fall or jump along the positions, past the 2^8 and 2^4 by which the kernel lets its maxima fall behind
    (heads in one and in two halves of an MMA's rows). Scores reach 28, so their fp32 rounding moves a probability by 2e-6. A probability
    times its V scale is a pair of halves relative to the largest V scale a warp has met, good to 2^-25 of that: where the order is
    random every warp meets the largest, and what counts has the smallest, so it spans 2^6 there (2^-19 of the result). The bound is
    that of the other cases."""
    S, nkv = 12 * 16 * 5 + 3, 2
    rng = np.random.default_rng(gqa + 7)
    at = np.arange(S) / S if ramp > 0 else 1 - np.arange(S) / S if ramp < 0 else rng.random(S)
    k8 = np.broadcast_to(rng.integers(-127, 128, (1, nkv, 128), dtype=np.int8), (S, nkv, 128)).copy()
    v8 = rng.integers(-127, 128, (S, nkv, 128), dtype=np.int8)
    q = synth.normal_f32(4300, nkv * gqa * 128).reshape(nkv, gqa, 128)
    dots = np.einsum("hgd,hd->hg", q.astype(np.float64), k8[0].astype(np.float64))
    q = (q / (dots[..., None] * 128 ** -0.5)).astype(np.float32)  # every head's score is the K scale
    ks = np.repeat((28 * at).astype(np.float32)[:, None], nkv, 1)
    vs = np.repeat((2.0 ** ((-20 if ramp else -6) * at)).astype(np.float32)[:, None] / 127, nkv, 1)
    want = oracle.attention_int8kv(q.reshape(-1), k8, v8, ks, vs, nkv * gqa, 128, nkv, S, gqa, 128 ** -0.5).reshape(-1, 128).astype(np.float64)
    out = torch.full((nkv * gqa * 128,), float("nan"), device="cuda")
    K.cuda_attention_int8kv(dev(q.reshape(-1)), dev(k8), dev(v8), dev(ks), dev(vs), out, nkv * gqa, 128, nkv, S, gqa, 128 ** -0.5)
    got = host(out).reshape(-1, 128).astype(np.float64)
    rel = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert rel.max() <= 2e-5, rel.max()


@pytest.mark.parametrize("V", [7, 256, 2049, 262144, 300001])
def test_sample_top_p_sizes(K, V):
    logits = (synth.normal_f32(4200 + V, V) * 2.0).astype(np.float32)
    d_l, res = dev(logits), torch.full((1,), -1, dtype=torch.int32, device="cuda")
    seeds = [int(s) for s in np.random.default_rng(V).integers(1, 2 ** 63, 12)]
    miss = 0
    for seed in seeds:
        K.cuda_sample_token(d_l, V, 0.8, 0.9, seed, res)
        miss += int(res.item()) != oracle.sample_top_p(logits, 0.8, 0.9, seed)
    assert miss <= 1, miss  # a cut or draw within float rounding of a boundary
