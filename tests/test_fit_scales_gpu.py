"""Operand scales of the FP16 fitting GEMMs: output units whose weights are
small beside the others' keep their accuracy, and rows of A far below one
static scale are off by no more than the pairs' resolution."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mdl(dpb):
    return importlib.import_module("deepmd_kit_lr_pt_b200.model")


def test_units_with_small_weights(dpb, mdl):
    """First layer with the units' weights 2^0 .. 2^-40 of the largest: the
    pre-activation error is within (2^-22 + 2^-23 * 100) sum |a| |b| of each
    unit's own terms (operand splits, and half an ulp of the truncating
    tensor-core sum per instruction of 16 k), and tanh adds 2^-22 of its
    value (2 ulp)."""
    cfg = mdl.SeAConfig()
    p = mdl.init_params(cfg, seed=5)
    rows, n = [130, 67], 197
    rng = np.random.default_rng(5)
    size = 2.0 ** -(np.arange(240) % 41)
    for f in p.fit:
        (W, b, d), *rest = f["layers"]
        f["layers"] = [((W * size).astype(np.float32), 0 * b, d), *rest]
    D = rng.normal(size=(n, 1600)).astype(np.float32)
    fit = mdl._FittingTC(p, rows, "cuda")
    scale = torch.full((n,), 2.0 ** 11, device="cuda")  # |D| < 8
    assert np.abs(D).max() < 8
    dD = torch.zeros((n, 1600), device="cuda")
    fit.layers(torch.tensor(D, device="cuda"), dD, row_scale=scale)
    got = fit.H1.cpu().numpy().astype(np.float64)
    o = 0
    for k, f in zip(rows, p.fit):
        W = f["layers"][0][0].astype(np.float64)
        a = D[o:o + k].astype(np.float64)
        want, mag = np.tanh(a @ W), np.abs(a) @ np.abs(W)
        err = np.abs(got[o:o + k] - want)
        assert (err <= (2.0 ** -22 + 2.0 ** -23 * 100) * mag + 2.0 ** -22 * np.abs(want)).all()
        o += k


@pytest.mark.parametrize("spread", [40, 9, 7, 0])
def test_units_of_uneven_weights(dpb, mdl, spread):
    """First layer with the units' weights 2^0 .. 2^-spread of the largest (a scale
    per row from a spread of 2^8 on): the
    pre-activation error is within (2^-22 + 2^-23 * 100) sum |a| |b| of each
    unit's own terms (operand splits, and half an ulp of the truncating
    tensor-core sum per instruction of 16 k), and tanh adds 2^-22 of its
    value (2 ulp)."""
    cfg = mdl.SeAConfig()
    p = mdl.init_params(cfg, seed=5)
    rows, n = [130, 67], 197
    rng = np.random.default_rng(5)
    size = 2.0 ** -(np.arange(240) % (spread + 1))
    for f in p.fit:
        (W, b, d), *rest = f["layers"]
        f["layers"] = [((W * size).astype(np.float32), 0 * b, d), *rest]
    D = rng.normal(size=(n, 1600)).astype(np.float32)
    fit = mdl._FittingTC(p, rows, "cuda")
    scale = torch.full((n,), 2.0 ** 11, device="cuda")  # |D| < 8
    assert np.abs(D).max() < 8
    dD = torch.zeros((n, 1600), device="cuda")
    if spread in (0, 40):  # the rows' largest entries differ by less than 2 by themselves
        assert all((t is not None) == (spread == 40) for t in fit.f16("1f")[1])
    fit.layers(torch.tensor(D, device="cuda"), dD, row_scale=scale)
    got = fit.H1.cpu().numpy().astype(np.float64)
    o = 0
    for k, f in zip(rows, p.fit):
        W = f["layers"][0][0].astype(np.float64)
        a = D[o:o + k].astype(np.float64)
        want, mag = np.tanh(a @ W), np.abs(a) @ np.abs(W)
        err = np.abs(got[o:o + k] - want)
        assert (err <= (2.0 ** -22 + 2.0 ** -23 * 100) * mag + 2.0 ** -22 * np.abs(want)).all()
        o += k


def test_batched_step_with_uneven_units(dpb):
    """The one-launch step takes the weights in the same form: forces and
    energies as the evaluator's, frame by frame. Both run the FP16 GEMMs, so
    what differs is the order of FP32 sums: 1e-5 of the largest."""
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    batch = importlib.import_module("deepmd_kit_lr_pt_b200.batch")
    coord, atype, box = wl.water_frame(3, seed=2)
    p = model.prepare(model.init_params(model.SeAConfig(), seed=2), coord, atype, box)
    for f in p.fit:
        f["layers"] = [(W * 2.0 ** -(np.arange(W.shape[1]) % 24), b, d)
                       for W, b, d in f["layers"]]
    e, f, _ = model.SeAEvaluator(p, atype, box).compute(coord)
    eb, fb, _ = batch.BatchEvaluator(p, [(coord, atype, box)] * 2).compute()
    n = atype.size
    for k in range(2):
        assert abs(eb[k] - e) <= 1e-5 * abs(e)
        assert np.abs(fb[k * n:(k + 1) * n] - f).max() <= 1e-5 * np.abs(f).max()


@pytest.mark.parametrize("N,K", [(80, 240), (240, 240), (1600, 240)])
def test_rows_below_a_static_scale(dpb, N, K):
    """Rows 2^0 .. 2^-24 below the bound that a_scale is made for, row_scale
    NULL. A scaled value v is held to max(2^-23 |v|, 2^-25): per entry
    (2^-22 + 2^-23 ceil(K / 16)) sum |a| |b| of relative errors and
    2^-25 / a_scale sum |b| of the absolute one."""
    cap = dpb._capi
    rng = np.random.default_rng(N)
    M = 150
    A = (rng.uniform(-1, 1, (M, K)) * 2.0 ** -(np.arange(M) % 25)[:, None]).astype(np.float32)
    B = (rng.normal(0, 1, (N, K)) * 2.0 ** -(np.arange(N) % 30)[:, None]).astype(np.float32)
    inv = 2.0 ** (np.ceil(np.log2(np.abs(B).max(1))) - 14)
    w = np.pad(B / inv[:, None], ((0, 0), (0, -K % 32)))
    hi = w.astype(np.float16)
    lo = (w - hi.astype(np.float64)).astype(np.float16)
    pairs = np.ascontiguousarray(np.stack([x.reshape(N, -1, 32) for x in (hi, lo)], 2))
    dev = lambda a: torch.tensor(np.asarray(a), device="cuda")  # noqa: E731
    Ad, Bd, bi = dev(A), dev(pairs), dev(inv.astype(np.float32))
    out = torch.full((M, N), float("nan"), device="cuda")
    status, e = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(M, device="cuda")
    a_scale, tr = np.array([2.0 ** 14], np.float32), np.array([M], np.int32)
    one = lambda t: (ctypes.c_void_p * 1)(t.data_ptr())  # noqa: E731
    s = torch.cuda.current_stream().cuda_stream
    cap.call("dpb_gemm_f16x3_rows_f32", cap.ptr(Ad), M, K, None, a_scale.ctypes.data, one(Bd),
             None, one(bi), N, tr.ctypes.data, 1, 0, cap.ptr(out), None, None, None, None, None,
             None, cap.ptr(e), cap.ptr(status), s)
    cap.call("dpb_status_check", cap.ptr(status), s)
    a, b = A.astype(np.float64), np.abs(B.astype(np.float64))
    tol = (2.0 ** -22 + 2.0 ** -23 * np.ceil(K / 16)) * (np.abs(a) @ b.T) + 2.0 ** -39 * b.sum(1)
    assert (np.abs(out.cpu().numpy() - a @ B.T.astype(np.float64)) <= tol).all()
