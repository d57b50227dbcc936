"""Helpers shared by the GPU parity tests (which call the kernels through the C ABI)."""
import numpy as np
import torch


def dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t: torch.Tensor) -> np.ndarray:
    return t.detach().cpu().numpy()


# Each output within 1e-3 relative L2 of the fp32 reference.
REL_L2_TOL = 1e-3


def assert_close_matvec(got: np.ndarray, want64: np.ndarray, abs_dot: np.ndarray | None = None, what=""):
    """Vector-level relative L2 <= 1e-3 against the fp64-accumulated oracle, plus a
    per-row bound |y - y_ref| <= 1e-3 * sum_c |w_rc x_c| when that scale is given."""
    got = got.astype(np.float64)
    assert np.all(np.isfinite(got)), f"{what}: non-finite output"
    denom = np.linalg.norm(want64)
    err = np.linalg.norm(got - want64)
    if denom > 0:
        assert err / denom <= REL_L2_TOL, f"{what}: rel L2 {err / denom:.3e} > {REL_L2_TOL}"
    else:
        assert err == 0
    if abs_dot is not None:
        bound = REL_L2_TOL * abs_dot + 1e-30
        worst = np.max(np.abs(got - want64) / bound)
        assert worst <= 1.0, f"{what}: per-row error {worst:.3e} x the 1e-3*sum|w x| bound"
    return err / denom if denom > 0 else 0.0


def layer_by_layer(model, l):
    """A layer by the kernels of their own that sharded models, and shapes outside the one-launch kernel, run."""
    import ctypes as C
    from mnemocuda_b200 import _lib
    from mnemocuda_b200 import kernels as K
    lib, d, ws, st = _lib.lib(), C.byref(model.desc), model.workspace.data_ptr(), K._stream(None)
    attn = torch.empty(model.cfg.q_dim, device="cuda")
    K._check(lib.mb200_decode_layer_attn(d, l, ws, model.pos.data_ptr(), attn.data_ptr(), st), "attention")
    K._check(lib.mb200_decode_layer_oproj(d, l, ws, attn.data_ptr(), model.hidden.data_ptr(), st), "O projection")
    K._check(lib.mb200_decode_layer_moe(d, l, ws, 1, model.hidden.data_ptr(), st), "experts")
