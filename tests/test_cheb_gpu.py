"""Descriptor passes on piecewise Chebyshev embeddings
(dpb_se_a_descriptor_{fwd,bwd}_cheb_f32) against the FP64 embedding net, over
the sizes where the groups of eight atoms, the channel tiles and the slot
chunks have edges, with unsorted rows, empty sections, padding and slots
outside the fitted range; and the host's expansion of a table."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

LO, HI = -1, 15


@pytest.fixture(scope="module")
def mods(dpb):
    return {m: importlib.import_module(f"deepmd_kit_lr_pt_b200.{m}")
            for m in ("_capi", "model", "table", "workload")}


def _model(mods, sel, M, ax):
    cfg = mods["workload"].SeAConfig(sel=sel, neuron=(M // 4, M // 2, M), axis_neuron=ax)
    p = mods["workload"].init_params(cfg, seed=M)
    nn = cfg.nnei
    p.davg = np.tile(np.array([0.06, 0, 0, 0]), (cfg.ntypes, nn))
    p.dstd = np.tile(np.array([0.11, 0.07, 0.07, 0.07]), (cfg.ntypes, nn))
    p.tables = mods["table"].build_tables(p.emb, p.davg, p.dstd, sel, 0.95, 0.5, 6.0)
    return p


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_expansion_matches_the_table(mods, seed):
    """Value within 1.5e-8 of the largest |G| at random points of the fitted
    range (the fit's own bound), and the FP16 pairs hold the coefficients to
    2^-22 of the largest."""
    p = _model(mods, (4,), 100, 16)
    p = mods["workload"].init_params(p.cfg, seed=seed)
    p.davg, p.dstd = np.tile([0.06, 0, 0, 0], (1, 4)), np.tile([0.11, 0.07, 0.07, 0.07], (1, 4))
    (table, info), = mods["table"].build_tables(p.emb, p.davg, p.dstd, (4,), 0.95, 0.5, 6.0)
    C, center, half, lut = mods["table"].chebyshev_net(table, info)
    x = np.random.default_rng(seed).uniform(info[0], info[1], 2000)
    r = lut[((x - info[0]) * mods["table"].CHEB_CELLS).astype(int)]
    t = (x - center[r]) / half[r]
    assert np.abs(t).max() <= 1 + 1e-12
    v = np.einsum("nk,nkm->nm", np.cos(np.arange(16) * np.arccos(np.clip(t, -1, 1))[:, None]),
                  C[r])
    G = mods["table"].embedding_derivatives(p.emb[0], x)[0]
    assert np.abs(v - G).max() <= 1.5e-8 * np.abs(G).max()
    fw, bw, scale = mods["table"].chebyshev_fragments(C)
    assert 2.0 ** round(np.log2(scale)) == scale and np.abs(C).max() * scale <= 2.0 ** 14
    h = fw.view(np.float16).astype(np.float64).reshape(*fw.shape[:3], 8)
    for lane in (0, 5, 31):
        for k, q in enumerate((0, 1, 8, 9)):
            j = np.arange(100) // 8
            m = np.arange(100)[np.arange(100) % 8 == lane >> 2]
            got = (h[..., k] + h[..., 4 + k])[:, j[m], lane] / scale
            want = C[:, 2 * (lane & 3) + q][:, m]
            assert np.abs(got - want).max() <= 2.0 ** -22 * np.abs(C).max()


def test_rough_nets_stay_on_the_table(mods):
    """A net too steep for 16 intervals, and bounds off the cell grid."""
    x = np.arange(LO, HI, 0.01)
    y = np.sin(60 * x)[:, None] * np.ones((1, 4))
    T = np.zeros((x.size + 600, 4, 6))
    T[:x.size, :, 0], T[:x.size, :, 1] = y, 60 * np.cos(60 * x)[:, None]
    info = np.array([LO, HI, 5 * HI, 0.01, 0.1, -1.0])
    assert mods["table"].chebyshev_net(T.reshape(-1, 24), info) is None
    bad = np.array([LO + 0.01, HI, 5 * HI, 0.01, 0.1, -1.0])
    assert mods["table"].chebyshev_net(T.reshape(-1, 24), bad) is None


def _rows(rng, n, sel, ordered):
    """Env rows: most x in the fitted range, a few below, above and beyond the
    tables, each section's tail empty."""
    em = np.zeros((n, sum(sel), 4), np.float32)
    o = 0
    for k in sel:
        for a in range(n):
            full = rng.integers(0, k + 1) if k else 0
            x = LO + 0.4 + rng.exponential(1.5, full)
            x[rng.random(full) < 0.02] = LO - 0.3
            x[rng.random(full) < 0.03] = HI + 20.0
            x[rng.random(full) < 0.01] = 5.0 * HI + 3.0
            x = np.sort(x)[::-1] if ordered else x
            em[a, o:o + full, 0] = x
            em[a, o:o + full, 1:] = rng.normal(0, 1, (full, 3))
            em[a, o + full:o + k, 0] = -0.06 / 0.11
        o += k
    return em


def _reference(mods, p, em, dD):
    """(xyz, D, net_deriv, scales) in FP64 from the quintic tables."""
    cfg, e = p.cfg, em.astype(np.float64)
    n, nn = e.shape[:2]
    G = np.zeros((n, nn, cfg.neuron[-1]))
    dG = np.zeros_like(G)
    for t, (a, b) in enumerate(zip(cfg.sec[:-1], cfg.sec[1:])):
        if b > a:
            lower, upper, mx, s0, s1 = p.tables[t][1][:5]
            T = p.tables[t][0].reshape(p.tables[t][0].shape[0], -1, 6)
            first = int(round((upper - lower) / s0))
            x = e[:, a:b, 0]
            xc = np.clip(x, lower, mx)
            fine = xc < upper
            row = np.where(fine, (xc - lower) / s0, first + (xc - upper) / s1)
            row = np.clip(row.astype(int), 0, T.shape[0] - 1)
            tt = (xc - np.where(fine, lower + row * s0, upper + (row - first) * s1))[..., None]
            c = T[row]
            v, g = c[..., 5], 5 * c[..., 5]
            for k in range(4, -1, -1):
                v = v * tt + c[..., k]
            for k in range(4, 0, -1):
                g = g * tt + k * c[..., k]
            G[:, a:b] = v + g * (x - xc)[..., None]
            dG[:, a:b] = g
    xyz = np.einsum("nsd,nsm->ndm", e, G) / nn
    D = np.einsum("ndm,nda->nma", xyz, xyz[:, :, :cfg.axis_neuron])
    dxyz = np.einsum("nma,nda->ndm", dD, xyz[:, :, :cfg.axis_neuron])
    dxyz[:, :, :cfg.axis_neuron] += np.einsum("nma,ndm->nda", dD, xyz)
    dxyz /= nn
    nd = np.einsum("ndm,nsm->nsd", dxyz, G)
    nd[..., 0] += np.einsum("ndm,nsm,nsd->ns", dxyz, dG, e)
    # the empty slots' sum at the first of them
    for a, b in zip(cfg.sec[:-1], cfg.sec[1:]):
        for i in range(n):
            empty = (e[i, a:b, 1:] == 0).all(-1) & (e[i, a:b, 0] == e[i, b - 1, 0] if b > a else 0)
            if empty.any():
                q = a + int(np.argmax(empty))
                nd[i, q], nd[i, q + 1:b] = nd[i, q:b].sum(0), 0.0
    s_xyz = np.einsum("nsd,nsm->ndm", np.abs(e), np.abs(G)).max() / nn
    s_nd = (np.einsum("ndm,nsm->nsd", np.abs(dxyz), np.abs(G)).max() * nn +
            np.einsum("ndm,nsm,nsd->ns", np.abs(dxyz), np.abs(dG), np.abs(e)).max())
    return xyz, D, nd, s_xyz, s_nd


@pytest.mark.gpu
@pytest.mark.parametrize("n,M,ax,sel,ordered", [
    (1, 100, 16, (46, 92), True), (7, 100, 16, (46, 92), True), (8, 8, 4, (3, 5), False),
    (9, 52, 4, (33, 0, 7), False), (33, 104, 16, (130,), True), (17, 128, 8, (32, 64, 1), False),
    (65, 100, 16, (31, 97, 60), False)])
@pytest.mark.parametrize("masked", [True, False])
def test_passes_match_fp64(mods, n, M, ax, sel, ordered, masked):
    """xyz, D and net_deriv; FP32 sums of up to sum(sel) slots and M channels
    and the 2^-22 of the split products, relative to the sums of magnitudes."""
    p = _model(mods, sel, M, ax)
    tabs = mods["model"].PipelineTables(p, "cuda:0", 3, n)
    assert tabs.nets is not None
    rng = np.random.default_rng(n)
    em = _rows(rng, n, sel, ordered)
    dD = rng.normal(0, 1, (n, M, ax)).astype(np.float32)
    xyz, D, nd, s_xyz, s_nd = _reference(mods, p, em, dD.astype(np.float64))
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    nan = lambda *s: torch.full(s, float("nan"), device="cuda")  # noqa: E731
    emd, dDd = dev(em), dev(dD[::-1].copy())
    drow = dev(np.arange(n, dtype=np.int32)[::-1].copy())
    gx, gD, gn = nan(n, 4, M), nan(n, M * ax), nan(n, sum(sel), 4)
    sec, s = p.cfg.sec, torch.cuda.current_stream().cuda_stream
    tabs.forward(gx, gD, drow, emd, sec, n, M, ax, s)
    if not masked:
        tabs.touched = None
    tabs.backward(gn, dDd, drow, gx, emd, sec, n, M, ax, s)
    eps = 2.0 ** -24 * (sum(sel) + 64)
    assert np.abs(gx.cpu().numpy() - xyz).max() <= eps * s_xyz
    got = gD.cpu().numpy()[::-1].reshape(n, M, ax)
    assert np.abs(got - D).max() <= 8 * eps * s_xyz * np.abs(xyz).max()
    assert np.abs(gn.cpu().numpy() - nd).max() <= 2.0 ** -24 * (M + sum(sel) + 64) * 4 * s_nd


@pytest.mark.gpu
def test_invalid_nets_are_refused(mods, dpb):
    p = _model(mods, (3, 5), 8, 4)
    tabs = mods["model"].PipelineTables(p, "cuda:0", 3, 4)
    x = torch.zeros(4 * 8 * 16, device="cuda")
    row = torch.zeros(4, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def run():
        tabs.forward(x, x, row, x, p.cfg.sec, 1, 8, 4, s)

    for field, value in (("nintervals", 17), ("nintervals", 0), ("fw", 0), ("lut", 0),
                         ("coef_scale", 0.0)):
        old = getattr(tabs.nets[1], field)
        setattr(tabs.nets[1], field, value)
        with pytest.raises(dpb._capi.DPBInvalidArgument):
            run()
        setattr(tabs.nets[1], field, old)
    assert ctypes.sizeof(mods["_capi"].ChebNet) == 56
