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


def _env(r, rmin, rmax):
    """env rows (s, s x / d, ...) of displacements r, s = sw(d) / d"""
    d = r.norm(dim=-1, keepdim=True)
    u = ((d - rmin) / (rmax - rmin)).clamp(0, 1)
    s = (u ** 3 * (-6 * u ** 2 + 15 * u - 10) + 1) / d
    return torch.cat([s, s * r / d], -1)


EDGES = [(1, (5,), 16), (2, (16, 17), 4), (9, (33, 1, 48), 16), (260, (20, 40), 16),
         (6, (15, 32, 3, 9), 8)]


def _tangent_and_gradients(dpb, n, sel, ax, dtype):
    """(kernel, FP64 autograd) pairs of xyz' and D' along a displacement field and
    of the gradients of <dD, D> + <dDt, D'> by every embedding weight"""
    cap = dpb._capi
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    cfg = wl.SeAConfig(sel=sel, axis_neuron=ax)
    p = wl.init_params(cfg, seed=n)
    nt, nn, M = len(sel), sum(sel), 100
    rmin, rmax = 1.5, 4.0
    rng = np.random.default_rng(n)
    grid = np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    dev = lambda a: torch.tensor(np.asarray(a), device="cuda")  # noqa: E731
    vp = lambda xs: (ctypes.c_void_p * len(xs))(*[x.data_ptr() for x in xs])  # noqa: E731
    x = dev(1.1 * grid + rng.uniform(-0.2, 0.2, (n, 3)))
    fbar, vbar = dev(rng.normal(0, 1, (n, 3))), dev(rng.normal(0, 0.3, (1, 3, 3)))
    ty = np.sort(rng.integers(0, nt, n)).astype(np.int32)
    avg, std = dev(rng.normal(0, .1, (nt, nn, 4))), dev(rng.uniform(.5, 1.5, (nt, nn, 4)))
    # one mean and deviation per section and column: pads of a section are alike
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
    lo = lambda q: q.detach().to(dtype).contiguous()  # noqa: E731
    suf = "f64" if dtype == torch.float64 else "f32"
    drow = np.arange(n, dtype=np.int32)[::-1].copy()
    Wl, bl, avg, std = [lo(q) for q in Ws], [lo(q) for q in bs], lo(avg), lo(std)
    dr, cw, box = dev(drow), x.contiguous(), dev(np.full((1, 3), 50.0))
    off, rf = dev(np.array([0, n], np.int32)), dev(np.zeros(n, np.int32))
    widths, sec = np.array([1, 25, 50, 100], np.int32), cfg.sec
    fold = np.ones(nt * nt, np.uint8)
    s = torch.cuda.current_stream().cuda_stream
    got_x = torch.full((n, 4, M), float("nan"), dtype=dtype, device="cuda")
    got_d = torch.full((n, M * ax), float("nan"), dtype=dtype, device="cuda")
    xc, xtc, nl, tyd = lo(xyz), lo(xyz_t), dev(packed), dev(ty)
    cap.call(f"dpb_se_a_train_tan_{suf}", cap.ptr(got_x), cap.ptr(got_d), cap.ptr(xc), cap.ptr(avg),
             cap.ptr(std), cap.ptr(fbar), cap.ptr(vbar), cap.ptr(cw), cap.ptr(nl), cap.ptr(tyd),
             cap.ptr(dr), cap.ptr(off), cap.ptr(box), cap.ptr(rf), 1, vp(Wl), vp(bl),
             widths.ctypes.data, sec.ctypes.data, sec.size, n, ax,
             ctypes.c_float(rmax), ctypes.c_float(rmin), s)
    g = [torch.zeros_like(q) for q in Wl + bl]
    scratch = torch.empty(8 * n * M, dtype=dtype, device="cuda")
    a1, a2 = lo(dD[dr.long()]), lo(dDt[dr.long()])
    cap.call(f"dpb_se_a_train_rev_{suf}", vp(g[:len(Ws)]), vp(g[len(Ws):]), cap.ptr(scratch),
             cap.ptr(xc), cap.ptr(xtc), cap.ptr(a1), cap.ptr(a2), cap.ptr(avg), cap.ptr(std),
             cap.ptr(fbar), cap.ptr(vbar), cap.ptr(cw), cap.ptr(nl), cap.ptr(tyd), cap.ptr(dr),
             cap.ptr(off), cap.ptr(box), cap.ptr(rf), 1, vp(Wl), vp(bl), widths.ctypes.data,
             sec.ctypes.data, sec.size, n, ax, fold.ctypes.data, ctypes.c_float(rmax),
             ctypes.c_float(rmin), s)
    return [(got_x, xyz_t.detach()), (got_d[dr.long()], Dt.detach())], list(zip(g, want))


def _errors(pairs):
    return [float((a.double() - b).abs().max()) / max(1.0, float(b.abs().max())) for a, b in pairs]


@pytest.mark.parametrize("n,sel,ax", EDGES)
def test_embedding_tangent_and_weight_gradients_match_autograd(dpb, n, sel, ax):
    """1e-12 of the largest for the tangents (100 x sum(sel) products), 1e-11 for
    the gradients, whose sums run over the atoms as well and cancel."""
    tangents, grads = _tangent_and_gradients(dpb, n, sel, ax, torch.float64)
    assert max(_errors(tangents)) <= 1e-12
    assert max(_errors(grads)) <= 1e-11


@pytest.mark.parametrize("n,sel,ax", EDGES)
def test_embedding_weight_gradients_fp32(dpb, n, sel, ax):
    """FP32: 2e-5 of the largest. Every factor (env row, tanh, adjoint) carries a
    few 6e-8, at most ten in a row, and the sums of up to 260 x 60 terms lose as
    many digits to cancellation as their terms exceed their total: a factor ten."""
    _, grads = _tangent_and_gradients(dpb, n, sel, ax, torch.float32)
    assert max(_errors(grads)) <= 2e-5
