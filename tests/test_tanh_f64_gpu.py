"""The tanh of the FP64 embedding passes, seen through the first layer of a net
whose other layers pass it on: xyz[1] of one neighbor with env row (x, 1, 0, 0)
is tanh(x w_c) for channel c."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _through_the_net(dpb, x, w):
    """tanh(x_i w_c) [n, 25] as the forward pass computes it"""
    cap = dpb._capi
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    cfg, n = wl.SeAConfig(sel=(1,), axis_neuron=4), x.size
    dev = lambda a: torch.tensor(np.asarray(a), device="cuda")  # noqa: E731
    vp = lambda xs: (ctypes.c_void_p * len(xs))(*[t.data_ptr() for t in xs])  # noqa: E731
    W = [dev(w.reshape(1, 25)), dev(np.zeros((25, 50))), dev(np.zeros((50, 100)))]
    b = [dev(np.zeros(k)) for k in (25, 50, 100)]
    em = np.zeros((n, 1, 4))
    em[:, 0, 0], em[:, 0, 1] = x, 1.0
    e, nl = dev(em), dev(np.full((n, 1), 27, np.int32))
    ty, dr = dev(np.zeros(n, np.int32)), dev(np.arange(n, dtype=np.int32))
    xyz = torch.full((n, 4, 100), float("nan"), dtype=torch.float64, device="cuda")
    D = torch.empty((n, 400), dtype=torch.float64, device="cuda")
    widths, sec, fold = np.array([1, 25, 50, 100], np.int32), cfg.sec, np.ones(1, np.uint8)
    cap.call("dpb_se_a_train_fwd_f64", cap.ptr(xyz), cap.ptr(D), cap.ptr(e), cap.ptr(nl),
             cap.ptr(ty), cap.ptr(dr), vp(W), vp(b), widths.ctypes.data, sec.ctypes.data,
             sec.size, n, 4, fold.ctypes.data, torch.cuda.current_stream().cuda_stream)
    out = xyz[:, 1].cpu().numpy()
    # the residual connections repeat the 25 channels four times
    assert np.array_equal(out[:, :25], out[:, 75:], equal_nan=True)
    return out[:, :25]


def test_error_bound(dpb):
    """Within 6 * 2^-53 of the value (the sum of its roundings) over 1e-300 .. 40,
    both signs, and densely where the power of two of exp(2 x) changes and around
    the clamp; against 64-bit mantissas on the host, and within that and CUDA's
    documented ulp (2^-52) of CUDA's own."""
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("needs an extended host precision")
    rng = np.random.default_rng(0)
    steps = (np.arange(0, 58) + 0.5) * np.log(2) / 2  # where k of 2 x = k ln 2 + r changes
    x = np.concatenate([10.0 ** rng.uniform(-300, 1.6, 4000), 10.0 ** rng.uniform(-9, 1.6, 20000),
                        (steps[:, None] * (1 + 1e-9 * rng.normal(size=(1, 60)))).ravel(),
                        rng.uniform(18, 22, 2000), 20 + np.arange(-50, 50) * 2.0 ** -48])
    w = 2.0 ** -np.arange(25.0) * np.where(np.arange(25) % 2, -1, 1)
    got = _through_the_net(dpb, x, w)
    arg = x[:, None] * w  # exact
    want = np.tanh(arg.astype(np.longdouble))
    err = np.abs((got - want) / want).astype(np.float64)
    print("worst", err.max() * 2.0 ** 53, "x 2^-53 at", arg.ravel()[err.argmax()])
    assert err.max() <= 6 * 2.0 ** -53
    cuda = torch.tanh(torch.tensor(arg, device="cuda")).cpu().numpy()
    print("CUDA's", float(np.abs((cuda - want) / want).max()) * 2.0 ** 53)
    assert (np.abs(got - cuda) <= (6 * 2.0 ** -53 + 2.0 ** -52) * np.abs(cuda)).all()


def test_special_values(dpb):
    w = np.where(np.arange(25) % 2, -1.0, 1.0)
    x = np.array([0.0, 5e-324, 1e-310, 2.3e-308, 19.0, 20.0, 20.5, 400.0, 1e300, np.inf, np.nan])
    got = _through_the_net(dpb, x, w)
    want = np.tanh(x)[:, None] * w
    assert (np.abs(got - want)[:-1] <= 2.0 ** -50 * np.abs(want)[:-1]).all()
    assert (np.abs(got[5:10]) == 1.0).all() and np.isnan(got[10]).all()
    assert (got[:4] == want[:4]).all()  # tiny arguments are returned as they are
