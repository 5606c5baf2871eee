"""tabulate_fusion_se_a and its gradients far beyond the table, where the linear
extrapolation is infinite or its powers overflow one by one: the results are
those of v + g delta, channel by channel."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LOWER, UPPER, MAX, S0, S1 = -1.0, 2.0, 6.0, 0.125, 0.5
ROWS = int((UPPER - LOWER) / S0 + (MAX - UPPER) / S1)


def _formula(T, x, dt):
    """value and slope [k, M] in the working type, as the reference forms them"""
    T = T.astype(dt)
    first = int((UPPER - LOWER) / S0)
    v, g = np.empty((x.size, T.shape[1]), dt), np.empty((x.size, T.shape[1]), dt)
    for s, xs in enumerate(x.astype(dt)):
        if xs < LOWER:
            r, t, d = 0, dt(0), xs - dt(LOWER)
        elif xs < MAX:
            r = int((xs - LOWER) / S0) if xs < UPPER else first + int((xs - UPPER) / S1)
            k = dt(LOWER + r * S0) if r < first else dt(UPPER + (r - first) * S1)
            t, d = xs - k, dt(0)
        else:
            r, t, d = ROWS - 1, dt(S1), xs - dt(MAX)
        c = T[r]
        g[s] = c[:, 1] + (2 * c[:, 2] + (3 * c[:, 3] + (4 * c[:, 4] + 5 * c[:, 5] * t) * t) * t) * t
        v[s] = c[:, 0] + (c[:, 1] + (c[:, 2] + (c[:, 3] + (c[:, 4] + c[:, 5] * t) * t) * t) * t) * t
        v[s] += g[s] * d
    return v, g


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("M", [6, 63, 64, 100, 130])
@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("far", [np.inf, -np.inf, 1e37, 3e20, -1e30, np.nan])
def test_far_extrapolation(dpb, dtype, M, far, own):
    """One slot at ``far`` among near ones (so no slot is folded). Infinite and
    NaN entries in the same places; the finite ones to 1e-4 (FP32) or 1e-12 of
    the terms' sizes (six powers, 34 slots, 130 channels)."""
    npt = np.dtype(dtype).type
    if dtype == "float64" and np.isfinite(far):
        far = np.sign(far) * abs(far) ** 8
    rng = np.random.default_rng(M)
    n, k, at = 3, 34, 20
    T = np.round(rng.normal(0, 1, (ROWS, M, 6)) * 64) / 64 * 0.5 ** np.arange(6)
    x = np.sort(rng.uniform(LOWER, MAX, (n, k)), 1)[:, ::-1].astype(npt).astype(np.float64)
    x[:, at] = far
    em = np.concatenate([x[..., None], rng.normal(0, 1, (n, k, 3))], -1).astype(npt)
    if not own:  # else the env row's first entry is x, as in a descriptor
        em[..., 0] = rng.normal(0, 1, (n, k))
    elif np.isfinite(far):
        pytest.skip("x times an extrapolation of its size overflows")
    dy, gx, ge = (rng.normal(0, 1, s).astype(npt) for s in ((n, 4, M), (n, k), (n, k, 4)))
    dev = lambda a: torch.tensor(np.asarray(a, npt), device="cuda")  # noqa: E731
    info = torch.tensor([LOWER, UPPER, MAX, S0, S1, -1.0], dtype=getattr(torch, dtype))
    table = dev(T.reshape(ROWS, -1))
    ops = torch.ops.deepmd
    out, = ops.tabulate_fusion_se_a(table, info, dev(x), dev(em), M)
    dx, de = ops.tabulate_fusion_se_a_grad(table, info, dev(x), dev(em), dev(dy), out)
    dz, = ops.tabulate_fusion_se_a_grad_grad(table, info, dev(x), dev(em), dev(gx), dev(ge), out,
                                             True)
    tol = 1e-4 if dtype == "float32" else 1e-12

    def check(got, want, mag):
        got = got.cpu().numpy().astype(np.float64).reshape(want.shape)
        assert (np.isnan(got) == np.isnan(want)).all()
        inf = np.isinf(want)
        assert (got[inf] == want[inf]).all() and not np.isinf(got[~inf & ~np.isnan(want)]).any()
        ok = np.isfinite(want)
        assert (np.abs(got - want)[ok] <= tol * mag[ok]).all()

    with np.errstate(all="ignore"):
        for i in range(n):
            v, g = (a.astype(np.float64) for a in _formula(T, x[i], npt))
            e, y = em[i].astype(np.float64), dy[i].astype(np.float64)
            a = np.abs
            big = np.where(np.isfinite(v), a(v), 0) + 4 * a(T).max() * (1 + a(x[i])[:, None])
            check(out[i], np.einsum("sd,sm->dm", e, v), np.einsum("sd,sm->dm", a(e), big))
            check(de[i], v @ y.T, big @ a(y).T)
            yg = e @ y
            gb = 24 * a(T).max() + a(g)
            check(dx[i], (g * yg).sum(1), (gb * (a(e) @ a(y))).sum(1))
            check(dz[i], np.einsum("sd,sm->dm", ge[i], v) +
                  np.einsum("s,sd,sm->dm", gx[i], e, g),
                  np.einsum("sd,sm->dm", a(ge[i]), big) +
                  np.einsum("s,sd,sm->dm", a(gx[i]), a(e), gb))
