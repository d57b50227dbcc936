"""The dense GEMM in each of its forms -- K split over a cluster, 64 / 128 / 256-token tiles, two CTAs on one tile -- at sizes
around their edges: rows past the last tile, an odd number of row tiles, K of one block and of a count the splits do not divide,
Q6_K tensors on an odd 2-byte address. Every token row against the C oracle."""
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


@pytest.mark.parametrize("kind", ["q4k", "q6k"])
@pytest.mark.parametrize("M,N,Kd", [(1, 1, 256), (9, 130, 2816), (65, 257, 4352), (63, 128, 8192), (100, 1377, 2048),
                                    (129, 2050, 512), (257, 8100, 256), (511, 8191, 768), (770, 5121, 256)])
def test_every_form(K, kind, M, N, Kd):
    gen, ref, call = ((synth.q4k_matrix, oracle.gemm_q4k_f16, K.mb200_gemm_q4k_f16) if kind == "q4k" else
                      (synth.q6k_matrix, oracle.gemm_q6k_f16, K.mb200_gemm_q6k_f16))
    w = gen(2700 + N, N, Kd)
    x = synth.normal_f16(2701 + M, M * Kd).reshape(M, Kd)
    want = ref(w, x, M, N, Kd).astype(np.float64)
    pad = 2 if kind == "q6k" else 16
    buf = torch.zeros(w.size + 32, dtype=torch.uint8, device="cuda")
    d_w = buf[pad:pad + w.size]
    d_w.copy_(dev(w))
    guard = torch.full((M * N + 64,), 7.0, device="cuda")
    out = guard[:M * N].view(M, N)
    for pdl in (False, True):
        before = K.mb200_set_pdl(pdl)
        out.fill_(float("nan"))
        call(d_w, dev(x), out, M, N, Kd)
        got = host(out).astype(np.float64)
        K.mb200_set_pdl(before)
        rel = np.linalg.norm(got - want, axis=1) / np.maximum(np.linalg.norm(want, axis=1), 1e-30)
        assert rel.max() <= 1e-3, (pdl, rel.max())
    assert bool((guard[M * N:] == 7.0).all())
    assert K.mb200_device_error() == 0


@pytest.mark.parametrize("kind,M,N,Kd", [("q6k", 1, 104, 256), ("q6k", 3, 100, 256), ("q6k", 17, 132, 512), ("q6k", 17, 130, 512),
                                         ("q6k", 33, 258, 1024), ("q6k", 65, 701, 2048), ("q6k", 16, 104, 768), ("q6k", 33, 104, 1280),
                                         ("q6k", 64, 104, 1536), ("q6k", 200, 1000, 1536), ("q4k", 16, 100, 768), ("q4k", 33, 100, 1280),
                                         ("q4k", 64, 100, 1536), ("q4k", 130, 1500, 1536)])
def test_rows_in_groups_and_splits(K, kind, M, N, Kd):
    """Q6_K on 16-byte addresses, where 8, 4, 2 or 1 rows at a time make a tensor map (K / 256 odd, 2, 4, 8), and with rows left over
    of that, which go the other way; K shared by 3, 5 and 6 CTAs. The bound is the one above (weights rounded to fp16 once: 2.8e-4)."""
    gen, ref, call = ((synth.q4k_matrix, oracle.gemm_q4k_f16, K.mb200_gemm_q4k_f16) if kind == "q4k" else
                      (synth.q6k_matrix, oracle.gemm_q6k_f16, K.mb200_gemm_q6k_f16))
    w = gen(2800 + N, N, Kd)
    x = synth.normal_f16(2801 + M, M * Kd).reshape(M, Kd)
    want = ref(w, x, M, N, Kd).astype(np.float64)
    guard = torch.full((M * N + 64,), 7.0, device="cuda")
    out = guard[:M * N].view(M, N)
    out.fill_(float("nan"))
    call(dev(w), dev(x), out, M, N, Kd)
    rel = np.linalg.norm(host(out).astype(np.float64) - want, axis=1) / np.linalg.norm(want, axis=1)
    assert rel.max() <= 1e-3, rel.max()
    assert bool((guard[M * N:] == 7.0).all())
    assert K.mb200_device_error() == 0


@pytest.mark.parametrize("kind,M,N,Kd", [
    # 64 tokens a tile, 8, 14, 6 and 5 super-blocks a CTA; rows 1, 4, 2 and 8 at a time
    ("q6k", 8, 8192, 4096), ("q6k", 30, 19000, 3584), ("q6k", 3, 6520, 3072), ("q6k", 1, 2480, 1280), ("q4k", 8, 8192, 4096),
    ("q6k", 68, 9632, 2048), ("q6k", 65, 4248, 2560), ("q6k", 100, 18944, 2304), ("q4k", 68, 9512, 2048),   # 128
    ("q6k", 700, 4100, 2048), ("q6k", 268, 6944, 1536), ("q6k", 265, 6440, 1280), ("q4k", 643, 3128, 1536),  # 256
    ("q6k", 512, 8192, 4096), ("q6k", 130, 9592, 3072), ("q6k", 257, 9472, 2816), ("q4k", 512, 8192, 4096),  # a pair
])
def test_weight_stages_used_again(K, kind, M, N, Kd):
    """More super-blocks a CTA than the ring of raw weights holds, in every form and, for Q6_K, every number of rows that make a tensor map. Rows
    repeat with a period that no tile divides. Against fp64 products of the weights rounded to fp16: what is left is fp32 accumulation (2e-5
    at 4096 columns) and weights that round to the other half (5e-6); a super-block taken before it is there would be 0.2."""
    gen, deq, call = ((synth.q4k_matrix, oracle.dequant_q4k, K.mb200_gemm_q4k_f16) if kind == "q4k" else
                      (synth.q6k_matrix, oracle.dequant_q6k, K.mb200_gemm_q6k_f16))
    n = min(N, 509)
    rows = np.arange(N) % n
    w = np.ascontiguousarray(gen(2900 + N, n, Kd).reshape(n, -1))
    w64 = dev(deq(w.reshape(-1), n, Kd).reshape(n, Kd)).half().double()
    d_w, x = dev(w[rows].reshape(-1)), dev(synth.normal_f16(2901 + M, M * Kd).reshape(M, Kd))
    assert d_w.data_ptr() % 16 == 0
    want = (x.double() @ w64.T)[:, torch.from_numpy(rows).cuda()]
    out = torch.empty(M, N, device="cuda")
    for pdl in (False, True):
        before = K.mb200_set_pdl(pdl)
        try:
            for _ in range(3):
                out.fill_(float("nan"))
                call(d_w, x, out, M, N, Kd)
                rel = (out.double() - want).norm(dim=1) / want.norm(dim=1)
                assert float(rel.max()) <= 1e-4, (pdl, float(rel.max()))
        finally:
            K.mb200_set_pdl(before)
    assert K.mb200_device_error() == 0
