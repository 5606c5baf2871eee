"""The training passes of embedding nets other than 25-50-100, which take the
general kernels: forward, force backward, tangent and weight gradients against
FP64 autograd, with one weight-gradient copy per block and per warp."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

from test_train_dmma_gpu import _env, _errors, _res

pytestmark = pytest.mark.gpu

NETS = [((8, 16, 32), 4, (20, 17)), ((10, 10, 20), 8, (33,)), ((25, 25, 100), 16, (9, 3, 16)),
        ((16, 40, 60), 16, (30, 21)), ((32, 64, 128), 16, (16, 33)), ((3, 5, 7), 5, (12, 40))]


def _all_passes(dpb, n, neuron, ax, sel, dtype):
    """(kernel, FP64 autograd) pairs: [xyz, D, dE/dR], [xyz', D'], gradients"""
    cap = dpb._capi
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    cfg = wl.SeAConfig(sel=sel, neuron=neuron, axis_neuron=ax)
    p = wl.init_params(cfg, seed=n)
    nt, nn, M = len(sel), sum(sel), neuron[-1]
    rmin, rmax = 1.5, 4.0
    rng = np.random.default_rng(n + M)
    grid = np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    dev = lambda a: torch.tensor(np.asarray(a), device="cuda")  # noqa: E731
    vp = lambda xs: (ctypes.c_void_p * len(xs))(*[x.data_ptr() for x in xs])  # noqa: E731
    x = dev(1.1 * grid + rng.uniform(-0.2, 0.2, (n, 3)))
    fbar, vbar = dev(rng.normal(0, 1, (n, 3))), dev(rng.normal(0, 0.3, (1, 3, 3)))
    ty = np.sort(rng.integers(0, nt, n)).astype(np.int32)
    avg, std = dev(rng.normal(0, .1, (nt, nn, 4))), dev(rng.uniform(.5, 1.5, (nt, nn, 4)))
    for a, b in zip(cfg.sec[:-1], cfg.sec[1:]):
        avg[:, a:b], std[:, a:b] = avg[:, a:a + 1].clone(), std[:, a:a + 1].clone()
    nb = np.full((n, nn), -1, np.int32)
    for i in range(n if n > 1 else 0):
        for a, b in zip(cfg.sec[:-1], cfg.sec[1:]):
            full = int(rng.integers(0, b - a + 1))
            nb[i, a:a + full] = (i + rng.integers(1, n, full)) % n
    packed = np.where(nb >= 0, nb * 27 + 13, -1).astype(np.int32)
    j, real = dev(np.maximum(nb, 0)).long(), dev(nb >= 0)[..., None]
    r = torch.where(real, x[j] - x[:, None], 1.0)
    w = torch.where(real, fbar[j] - fbar[:, None] + r @ vbar[0].T, 0.0)
    R, Rd = torch.func.jvp(lambda q: _env(q, rmin, rmax), (r,), (w,))
    tl = dev(ty).long()
    R = (torch.where(real, R, 0.0) - avg[tl]) / std[tl]
    Rd = -torch.where(real, Rd, 0.0) / std[tl]  # the env derivative is by the center atom
    Ws = [dev(W) for net in p.emb for W, _ in net]
    bs = [dev(b) for net in p.emb for _, b in net]
    leaf = [q.clone().requires_grad_() for q in Ws + bs]

    def xyz_of(R):
        out = 0
        for t, (a, b) in enumerate(zip(cfg.sec[:-1], cfg.sec[1:])):
            h = R[:, a:b, :1]
            for k in range(3):
                W, bias = leaf[3 * t + k], leaf[len(Ws) + 3 * t + k]
                y = torch.tanh(h @ W + bias)
                h = _res(W, h, y) if k else y
            out = out + R[:, a:b].transpose(1, 2) @ h
        return out / nn

    def D_of(X):
        return (X.transpose(1, 2) @ X[:, :, :ax]).reshape(n, -1)

    xyz, xyz_t = torch.func.jvp(xyz_of, (R,), (Rd,))
    D, Dt = torch.func.jvp(D_of, (xyz,), (xyz_t,))
    dD, dDt = (dev(rng.normal(0, 1, (n, M * ax))) for _ in range(2))
    want = torch.autograd.grad((D * dD).sum() + (Dt * dDt).sum(), leaf)
    Rl = R.clone().requires_grad_()
    gR, = torch.autograd.grad((D_of(xyz_of(Rl)) * dD).sum(), Rl)
    lo = lambda q: q.detach().to(dtype).contiguous()  # noqa: E731
    suf = "f64" if dtype == torch.float64 else "f32"
    dr = dev(np.arange(n, dtype=np.int32)[::-1].copy())
    Wl, bl, avg, std = [lo(q) for q in Ws], [lo(q) for q in bs], lo(avg), lo(std)
    off, rf = dev(np.array([0, n], np.int32)), dev(np.zeros(n, np.int32))
    box = dev(np.full((1, 3), 50.0))
    widths, sec = np.array([1, *neuron], np.int32), cfg.sec
    fold = np.ones(nt * nt, np.uint8)
    s = torch.cuda.current_stream().cuda_stream
    new = lambda *shape: torch.full(shape, float("nan"), dtype=dtype, device="cuda")  # noqa: E731
    P = cap.ptr
    em, nl, tyd = lo(R), dev(packed), dev(ty)
    gx, gD, ge, xb = new(n, 4, M), new(n, M * ax), new(n, nn, 4), new(n, 4, M)
    net = (vp(Wl), vp(bl), widths.ctypes.data, sec.ctypes.data, sec.size, n, ax)
    a1, a2 = lo(dD[dr.long()]), lo(dDt[dr.long()])
    cap.call(f"dpb_se_a_train_fwd_{suf}", P(gx), P(gD), P(em), P(nl), P(tyd), P(dr), *net,
             fold.ctypes.data, s)
    cap.call(f"dpb_se_a_train_bwd_{suf}", P(ge), P(xb), P(em), P(gx), P(a1), P(nl), P(tyd), P(dr),
             *net, s)
    tx, tD = new(n, 4, M), new(n, M * ax)
    geom = (P(avg), P(std), P(fbar), P(vbar), P(x), P(nl), P(tyd), P(dr), P(off), P(box), P(rf), 1)
    rc, rs = ctypes.c_float(rmax), ctypes.c_float(rmin)
    xc, xtc = lo(xyz), lo(xyz_t)
    cap.call(f"dpb_se_a_train_tan_{suf}", P(tx), P(tD), P(xc), *geom, *net, rc, rs, s)
    g = [torch.zeros_like(q) for q in Wl + bl]
    scratch = torch.empty(8 * n * M, dtype=dtype, device="cuda")
    cap.call(f"dpb_se_a_train_rev_{suf}", vp(g[:len(Ws)]), vp(g[len(Ws):]), P(scratch), P(xc),
             P(xtc), P(a1), P(a2), *geom, *net, fold.ctypes.data, rc, rs, s)
    m = dev(nb >= 0)
    first = [(gx, xyz.detach()), (gD[dr.long()], D.detach())]
    if bool(m.any()):
        first.append((ge[m], gR[m]))
    return (first, [(tx, xyz_t.detach()), (tD[dr.long()], Dt.detach())], list(zip(g, want)))


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("shared_acc", [0, 1])
@pytest.mark.parametrize("neuron,ax,sel", NETS)
@pytest.mark.parametrize("n", [1, 9, 150])
def test_general_nets(dpb, neuron, ax, sel, n, shared_acc, dtype):
    """FP64: 1e-12 of the largest for values and tangents (sums of up to 128 x 50
    products), 1e-11 for the gradients, whose sums run over the atoms and cancel.
    FP32: factors of a few 6e-8, at most ten in a row, and a factor ten for the
    cancellation: 2e-5."""
    at = importlib.import_module("deepmd_kit_lr_pt_b200.autotune")
    old = at.get("train_rev_shared_acc")
    at.set_knob("train_rev_shared_acc", shared_acc)
    try:
        first, tangents, grads = _all_passes(dpb, n, neuron, ax, sel, getattr(torch, dtype))
    finally:
        at.set_knob("train_rev_shared_acc", old)
    f64 = dtype == "float64"
    assert max(_errors(first)) <= (1e-12 if f64 else 2e-5)
    assert max(_errors(tangents)) <= (1e-12 if f64 else 2e-5)
    assert max(_errors(grads)) <= (1e-11 if f64 else 2e-5)
