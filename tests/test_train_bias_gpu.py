"""The FP32 tangent and reverse passes on the matrix instructions carry no
systematic error: their results are not shrunk against FP64 on the same inputs."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(dpb, dt, n, sel, ax, cfg, d):
    cap = dpb._capi
    M, suf, nt = 100, ("f64" if dt == torch.float64 else "f32"), len(sel)
    dev = lambda a: torch.tensor(np.asarray(a), device="cuda")  # noqa: E731
    lo = lambda a: dev(a).to(dt).contiguous()  # noqa: E731
    vp = lambda xs: (ctypes.c_void_p * len(xs))(*[x.data_ptr() for x in xs])  # noqa: E731
    p = cap.ptr
    W, b = [lo(q) for q in d["W"]], [lo(q) for q in d["b"]]
    avg, std, x, xt, a1, a2 = (lo(d[k]) for k in ("avg", "std", "xyz", "xyzt", "dD", "dDt"))
    fb, vb, cw, box = dev(d["fbar"]), dev(d["vbar"]), dev(d["x"]), dev(np.full((1, 3), 50.0))
    nl, ty, dr = dev(d["packed"]), dev(d["ty"]), dev(np.arange(n, dtype=np.int32))
    off, rf = dev(np.array([0, n], np.int32)), dev(np.zeros(n, np.int32))
    wid, sec, fold = np.array([1, 25, 50, 100], np.int32), cfg.sec, np.ones(nt * nt, np.uint8)
    s = torch.cuda.current_stream().cuda_stream
    out = [torch.zeros((n, 4, M), dtype=dt, device="cuda"),
           torch.zeros((n, M * ax), dtype=dt, device="cuda")]
    g = [torch.zeros_like(q) for q in W + b]
    scratch = torch.empty(8 * n * M, dtype=dt, device="cuda")
    geom = (p(avg), p(std), p(fb), p(vb), p(cw), p(nl), p(ty), p(dr), p(off), p(box), p(rf), 1)
    rc, rs = ctypes.c_float(6.0), ctypes.c_float(0.5)
    cap.call(f"dpb_se_a_train_tan_{suf}", p(out[0]), p(out[1]), p(x), *geom, vp(W), vp(b),
             wid.ctypes.data, sec.ctypes.data, sec.size, n, ax, rc, rs, s)
    cap.call(f"dpb_se_a_train_rev_{suf}", vp(g[:len(W)]), vp(g[len(W):]), p(scratch), p(x), p(xt),
             p(a1), p(a2), *geom, vp(W), vp(b), wid.ctypes.data, sec.ctypes.data, sec.size, n, ax,
             fold.ctypes.data, rc, rs, s)
    return [q.double() for q in out + g]


def _shift(dpb, seed):
    """<got - want, want> / <want, want> of xyz', D' and each weight gradient."""
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    n, sel, ax = 300, (46, 92), 16
    cfg = wl.SeAConfig(sel=sel, axis_neuron=ax)
    par = wl.init_params(cfg, seed=seed)
    rng = np.random.default_rng(seed)
    r32 = lambda a: np.asarray(a, np.float32).astype(np.float64)  # noqa: E731
    grid = np.stack(np.meshgrid(*[np.arange(7)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    nn, nt = sum(sel), len(sel)
    avg, std = r32(rng.normal(0, .1, (nt, nn, 4))), r32(rng.uniform(.5, 1.5, (nt, nn, 4)))
    nb = np.full((n, nn), -1, np.int32)
    for a, b in zip(cfg.sec[:-1], cfg.sec[1:]):
        avg[:, a:b], std[:, a:b] = avg[:, a:a + 1], std[:, a:a + 1]
        for i in range(n):
            full = int(rng.integers((b - a) // 2, b - a + 1))
            nb[i, a:a + full] = (i + 1 + rng.permutation(n - 1)[:full]) % n
    d = {"x": 1.1 * grid + rng.uniform(-.2, .2, (n, 3)), "fbar": rng.normal(0, 1, (n, 3)),
         "vbar": rng.normal(0, .3, (1, 3, 3)), "avg": avg, "std": std,
         "packed": np.where(nb >= 0, nb * 27 + 13, -1).astype(np.int32),
         "ty": np.sort(rng.integers(0, nt, n)).astype(np.int32),
         "W": [r32(W) for net in par.emb for W, _ in net],
         "b": [r32(b) for net in par.emb for _, b in net],
         "xyz": r32(rng.normal(0, .3, (n, 4, 100))), "xyzt": r32(rng.normal(0, .3, (n, 4, 100))),
         "dD": r32(rng.normal(0, 1, (n, 100 * ax))), "dDt": r32(rng.normal(0, 1, (n, 100 * ax)))}
    got, want = (_run(dpb, dt, n, sel, ax, cfg, d) for dt in (torch.float32, torch.float64))
    return [float(((a - b) * b).sum() / (b * b).sum()) for a, b in zip(got, want)]


def test_no_systematic_shrinking(dpb):
    """Rounded FP32 sums leave each draw of inputs a factor of either sign (of
    order 2^-25 for the weight gradients, whose entries share their roundings; plain
    FMA kernels show the same), truncated ones add one of the same sign to every
    draw, 2^-25 and more per product of a layer. So the mean over 16 draws is held: to
    2^-26 for xyz' and D' (30,000 and 480,000 entries a draw), to 2^-25 for the mean
    of the weight gradients."""
    shift = np.array([_shift(dpb, seed) for seed in range(16)])
    mean = shift.mean(axis=0)
    assert np.abs(mean[:2]).max() <= 2.0 ** -26, shift
    assert abs(mean[2:].mean()) <= 2.0 ** -25, shift
