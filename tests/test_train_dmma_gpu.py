"""The FP64 embedding passes of the standard net (forward and force backward)
at the edges of their 16-row groups and of the CTA splits, against FP64
autograd; four neighbor types take the general kernels on the same inputs."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _res(W, x, y):
    return y + (x if W.shape[0] == W.shape[1] else
                torch.cat([x, x], -1) if W.shape[1] == 2 * W.shape[0] else 0)


@pytest.mark.parametrize("n,sel,ax", [(1, (5,), 16), (3, (16, 17), 4), (7, (33, 1, 48), 16),
                                      (301, (20, 40), 16), (5, (15, 32, 3, 9), 8)])
def test_embedding_passes_match_autograd(dpb, n, sel, ax):
    """xyz, D and dE/d(em) of E = <dD, D> to 1e-12 of their largest (sums of at
    most 100 x sum(sel) products, each tanh within a few 1e-16)."""
    cap = dpb._capi
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    cfg = wl.SeAConfig(sel=sel, axis_neuron=ax)
    p = wl.init_params(cfg, seed=n)
    nt, nn, M = len(sel), sum(sel), 100
    rng = np.random.default_rng(n)
    em = np.zeros((n, nn, 4))
    nlist = np.full((n, nn), -1, np.int32)
    for i in range(n):
        for a, b in zip(cfg.sec[:-1], cfg.sec[1:]):
            full = int(rng.integers(0, b - a + 1))
            em[i, a:a + full] = rng.normal(0, 1, (full, 4)) * [3, 1, 1, 1]
            em[i, a + full:b, 0] = -0.5
            nlist[i, a:a + full] = 27
    dD = rng.normal(0, 1, (n, M * ax))
    dev = lambda a: torch.tensor(np.asarray(a), device="cuda")  # noqa: E731
    vp = lambda xs: (ctypes.c_void_p * len(xs))(*[x.data_ptr() for x in xs])  # noqa: E731
    Ws = [dev(W) for net in p.emb for W, _ in net]
    bs = [dev(b) for net in p.emb for _, b in net]
    e = dev(em).requires_grad_()
    xyz = 0
    for t, (a, b) in enumerate(zip(cfg.sec[:-1], cfg.sec[1:])):
        h = e[:, a:b, :1]
        for k in range(3):
            W = Ws[3 * t + k]
            h = _res(W, h, torch.tanh(h @ W + bs[3 * t + k])) if k else \
                torch.tanh(h @ W + bs[3 * t])
        xyz = xyz + e[:, a:b].transpose(1, 2) @ h
    xyz = xyz / nn
    D = (xyz.transpose(1, 2) @ xyz[:, :, :ax]).reshape(n, -1)
    g, = torch.autograd.grad((D * dev(dD)).sum(), e)
    drow = np.arange(n, dtype=np.int32)[::-1].copy()
    out = [torch.full(s, float("nan"), dtype=torch.float64, device="cuda")
           for s in ((n, 4, M), (n, M * ax), (n, nn, 4), (n, 4, M))]
    ty, nl, dr = dev(np.zeros(n, np.int32)), dev(nlist), dev(drow)
    widths, sec = np.array([1, 25, 50, 100], np.int32), cfg.sec
    fold = np.ones(nt * nt, np.uint8)
    s = torch.cuda.current_stream().cuda_stream
    em_d, dDr = dev(em), dev(dD[drow])
    cap.call("dpb_se_a_train_fwd_f64", cap.ptr(out[0]), cap.ptr(out[1]), cap.ptr(em_d),
             cap.ptr(nl), cap.ptr(ty), cap.ptr(dr), vp(Ws), vp(bs), widths.ctypes.data,
             sec.ctypes.data, sec.size, n, ax, fold.ctypes.data, s)
    cap.call("dpb_se_a_train_bwd_f64", cap.ptr(out[2]), cap.ptr(out[3]), cap.ptr(em_d),
             cap.ptr(out[0]), cap.ptr(dDr), cap.ptr(nl), cap.ptr(ty), cap.ptr(dr), vp(Ws), vp(bs),
             widths.ctypes.data, sec.ctypes.data, sec.size, n, ax, s)
    real = dev(nlist) >= 0
    for got, want in ((out[0], xyz), (out[1][dev(drow).long()], D), (out[2][real], g[real])):
        if want.numel():
            got, want = got.detach(), want.detach()
            assert float((got - want).abs().max()) <= 1e-12 * max(1.0, float(want.abs().max()))
    assert bool((out[2][~real] == 0).all())
