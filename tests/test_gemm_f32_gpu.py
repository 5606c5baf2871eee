"""dpb_gemm_f32, the GEMM of FP32 layers whose width the tensor-core tiles do not
divide: both tile shapes, every transpose, edges, bias and accumulation."""

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (63, 65, 17), (127, 60, 200), (128, 64, 8),
                                   (129, 65, 33), (300, 130, 7), (1000, 50, 0), (257, 1, 90)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("with_bias,accumulate", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_matches_fp64(dpb, big, M, N, K, ta, tb, with_bias, accumulate):
    """Per entry within 2^-24 (K + 2) (sum |a| |b| + |bias| + |c|): one rounding per
    product and addition of an FP32 sum in any order."""
    cap = dpb._capi
    at = importlib.import_module("deepmd_kit_lr_pt_b200.autotune")
    rng = np.random.default_rng(M * 7 + N * 3 + K)
    A, B = (rng.normal(0, 1, s).astype(np.float32) for s in ((M, K), (K, N)))
    bias, C = (rng.normal(0, 1, s).astype(np.float32) for s in ((N,), (M, N)))
    # leading dimensions beyond the rows, as views of wider arrays have them
    pad = lambda a: np.pad(a, ((0, 0), (0, 3)), constant_values=np.nan)  # noqa: E731
    Am, Bm = pad(A.T if ta else A), pad(B.T if tb else B)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    Ad, Bd, Cd, bd = dev(Am), dev(Bm), dev(pad(C)), dev(bias)
    old = at.get("gemm_simt_big")
    at.set_knob("gemm_simt_big", big)
    try:
        cap.call("dpb_gemm_f32", cap.ptr(Cd), cap.ptr(Ad), cap.ptr(Bd),
                 cap.ptr(bd) if with_bias else None, M, N, K, Am.shape[1], Bm.shape[1], N + 3, ta,
                 tb, accumulate, torch.cuda.current_stream().cuda_stream)
    finally:
        at.set_knob("gemm_simt_big", old)
    a, b = A.astype(np.float64), B.astype(np.float64)
    want, mag = a @ b, np.abs(a) @ np.abs(b)
    if with_bias:
        want, mag = want + bias, mag + np.abs(bias)
    if accumulate:
        want, mag = want + C, mag + np.abs(C)
    got = Cd.cpu().numpy()
    assert np.isnan(got[:, N:]).all()  # nothing written beyond the row
    assert (np.abs(got[:, :N] - want) <= 2.0 ** -24 * (K + 2) * mag).all()
