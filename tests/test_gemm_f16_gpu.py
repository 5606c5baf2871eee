"""The split-FP16 tensor-core GEMM (dpb_gemm_f16x3_f32) against FP64: edges of
the row tiles, of the k-blocks and of the column tiles, chunked and whole
accumulation, and rows of very different size (their scales)."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pairs(B, scale):
    """[N, KB, 2, 32] halves of B * scale (dpb_gemm_f16x3_f32's layout)."""
    w = np.pad(B * scale, ((0, 0), (0, -B.shape[1] % 32)))
    hi = w.astype(np.float16)
    lo = (w - hi.astype(np.float64)).astype(np.float16)
    return np.ascontiguousarray(np.stack([x.reshape(B.shape[0], -1, 32) for x in (hi, lo)], 2))


@pytest.mark.parametrize("rows,N,K", [((1,), 80, 4), ((127, 2), 240, 240), ((128, 0, 129), 160, 32),
                                      ((300, 5), 240, 1600), ((64,), 1600, 240),
                                      ((257, 130), 80, 292)])
def test_matches_fp64(dpb, rows, N, K):
    """|C - A B^T| <= (2^-22 + 2^-23 ceil(K / 16)) sum |a| |b| per entry: each
    operand's split to 2^-23 and the lo lo product, and the tensor cores'
    truncating FP32 sum of K / 16 instructions times three products, half an
    ulp each on average."""
    cap = dpb._capi
    rng = np.random.default_rng(K + N)
    M, nt = sum(rows), len(rows)
    A = rng.normal(0, 1, (M, K)) * 10.0 ** rng.integers(-12, 13, (M, 1))
    A = A.astype(np.float32)
    B = [rng.normal(0, K ** -0.5, (N, K)).astype(np.float32) for _ in rows]
    big = np.abs(A).max(1)
    rs = (2.0 ** (13 - np.ceil(np.log2(big)))).astype(np.float32)
    bs = np.array([2.0 ** (14 - np.ceil(np.log2(np.abs(b).max()))) for b in B], np.float32)
    keep = [torch.tensor(_pairs(b.astype(np.float64), s), device="cuda") for b, s in zip(B, bs)]
    bp = (ctypes.c_void_p * nt)(*[t.data_ptr() for t in keep])
    out = torch.full((M, N), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    e = torch.zeros(max(M, 1), device="cuda")
    tr = np.array(rows, np.int32)
    one = np.full(nt, 2.0, np.float32)  # with the row scales: 2^14
    Ad, rd = torch.tensor(A, device="cuda"), torch.tensor(rs, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    cap.call("dpb_gemm_f16x3_f32", cap.ptr(Ad), M, K, cap.ptr(rd), one.ctypes.data, bp,
             bs.ctypes.data, N, tr.ctypes.data, nt, 0, cap.ptr(out), None, None, None, None, None,
             None, cap.ptr(e), cap.ptr(status), s)
    cap.call("dpb_status_check", cap.ptr(status), s)
    got = out.cpu().numpy().astype(np.float64)
    tol = 2.0 ** -22 + 2.0 ** -23 * np.ceil(K / 16)
    o = 0
    for n, b in zip(rows, B):
        a = A[o:o + n].astype(np.float64)
        ref, mag = a @ b.T.astype(np.float64), np.abs(a) @ np.abs(b.T).astype(np.float64)
        assert (np.abs(got[o:o + n] - ref) <= tol * mag).all()
        o += n


def test_evaluator_scales_hold_for_large_weights(dpb):
    """Operand bounds of the fitting layers: with weights 30 times the usual
    the FP16 path still agrees with the TF32 path (fit_split_b = 1)."""
    import importlib

    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    mdl = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    at = importlib.import_module("deepmd_kit_lr_pt_b200.autotune")
    coord, atype, box = wl.water_frame(3, seed=1)
    p = mdl.prepare(mdl.init_params(mdl.SeAConfig(), seed=1), coord, atype, box)
    for f in p.fit:
        f["layers"] = [(W * 30.0, b, d) for W, b, d in f["layers"]]
        f["out"] = (f["out"][0] * 1e3, f["out"][1])
    ev = mdl.SeAEvaluator(p, atype, box)
    assert ev.ptab.row_scale is not None
    e0, f0, v0 = ev.compute(coord)
    ev.check()
    at.set_knob("fit_split_b", 1)
    try:
        e1, f1, v1 = ev.compute(coord)
    finally:
        at.set_knob("fit_split_b", 0)
    assert np.isfinite(f0).all() and abs(e0 - e1) <= 1e-5 * abs(e1)
    assert np.abs(f0 - f1).max() <= 2e-4 * np.abs(f1).max()
