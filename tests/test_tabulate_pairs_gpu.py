"""tabulate_fusion_se_a and its two gradients at the edges of the 64-channel
blocks, of the 32-slot chunks and of the wide row loads (odd channel counts,
tables off the 16-byte boundary), against the FP64 formulas."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LOWER, UPPER, MAX, S0, S1 = -1.0, 2.0, 6.0, 0.125, 0.5
ROWS = int((UPPER - LOWER) / S0 + (MAX - UPPER) / S1)


def _poly(T, x):
    """Value and slope [n, k, M] with the linear tails."""
    xc = np.clip(x, LOWER, MAX)
    first = int((UPPER - LOWER) / S0)
    r = np.where(xc < UPPER, (xc - LOWER) / S0, first + (xc - UPPER) / S1).astype(int)
    r = np.clip(r, 0, ROWS - 1)
    t = (xc - np.where(r < first, LOWER + r * S0, UPPER + (r - first) * S1))[..., None]
    c = T[r]
    v = sum(c[..., k] * t ** k for k in range(6))
    g = sum(k * c[..., k] * t ** (k - 1) for k in range(1, 6))
    return v + g * (x - xc)[..., None], g


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,k,M,shift", [(1, 1, 1, 0), (5, 31, 2, 0), (3, 32, 63, 0),
                                         (4, 33, 64, 1), (2, 130, 65, 0), (7, 92, 100, 0),
                                         (3, 64, 128, 1), (1, 40, 129, 0), (2, 5, 1024, 0),
                                         (2500, 3, 6, 0)])
def test_matches_fp64_formulas(dpb, dtype, n, k, M, shift):
    """Per entry, |error| <= 2^-p (terms + 16) sum |terms|, p = 24 or 53, of
    sums of k slots x 6 powers (forward, grad_grad) or M channels x 6 (grad)."""
    eps = 2.0 ** (-24 if dtype == "float32" else -53)
    rng = np.random.default_rng(100 * M + k)
    npt = np.dtype(dtype)
    T = rng.normal(0, 1, (ROWS, M, 6)).astype(npt).astype(np.float64)
    x = np.sort(rng.uniform(LOWER - 0.5, MAX + 0.5, (n, k)), 1)[:, ::-1]
    x = np.round(x * 1024) / 1024  # exact in FP32, as are the strides
    em = np.concatenate([x[..., None], rng.normal(0, 1, (n, k, 3))], -1)
    full = rng.integers(0, k + 1, n)
    for i in range(n):
        em[i, full[i]:, 0], em[i, full[i]:, 1:] = -0.75, 0.0
    em = em.astype(npt).astype(np.float64)
    dy, gx, ge = (rng.normal(0, 1, s).astype(npt).astype(np.float64)
                  for s in ((n, 4, M), (n, k), (n, k, 4)))
    v, g = _poly(T, em[..., 0])
    # the empty slots count once, at the first of them, times their number
    w = np.ones((n, k))
    for i in range(n):
        if full[i] < k:
            w[i, full[i]], w[i, full[i] + 1:] = k - full[i], 0.0

    def dev(a, off=0):
        buf = torch.zeros(a.size + 4, dtype=getattr(torch, dtype), device="cuda")
        out = buf[off:off + a.size].view(a.shape)
        out.copy_(torch.tensor(a))
        return out

    # FP32 tables may start on any 8-byte boundary
    table = dev(T.reshape(ROWS, -1), 2 * shift if dtype == "float32" else 0)
    info = torch.tensor([LOWER, UPPER, MAX, S0, S1, -1.0], dtype=getattr(torch, dtype))
    e, ex = dev(em), dev(em[..., 0].copy())
    out, = torch.ops.deepmd.tabulate_fusion_se_a(table, info, ex, e, M)
    dx, de = torch.ops.deepmd.tabulate_fusion_se_a_grad(table, info, ex, e, dev(dy), out)
    dz, = torch.ops.deepmd.tabulate_fusion_se_a_grad_grad(table, info, ex, e, dev(gx), dev(ge),
                                                          out, True)
    av, ag = (np.abs(a) + 4 * np.abs(T).max() for a in (v, g))  # the powers' own terms

    def check(got, want, mag, terms):
        err = np.abs(got.cpu().numpy().astype(np.float64) - want)
        assert (err <= eps * (terms + 16) * (mag + 1e-30)).all(), float((err / mag).max() / eps)

    def slots(a, b):
        return np.einsum("ns,nsd,nsm->ndm", w, a, b)

    check(out, slots(em, v), slots(np.abs(em), av), 6 * k)
    dyg = np.einsum("nsd,ndm->nsm", em, dy)
    check(dx, w * np.einsum("nsm,nsm->ns", g, dyg),
          w * np.einsum("nsm,nsd,ndm->ns", ag, np.abs(em), np.abs(dy)), 6 * M)
    check(de, w[..., None] * np.einsum("nsm,ndm->nsd", v, dy),
          w[..., None] * np.einsum("nsm,ndm->nsd", av, np.abs(dy)), 6 * M)
    check(dz, slots(ge, v) + slots(gx[..., None] * em, g),
          slots(np.abs(ge), av) + slots(np.abs(gx[..., None] * em), ag), 12 * k)
