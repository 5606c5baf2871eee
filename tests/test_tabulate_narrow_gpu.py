"""tabulate_fusion_se_a and its gradients at the widths where the kernel changes
(32-channel blocks, grad_grad by channels), few and many atoms: every route
against the formulas in FP64."""

import numpy as np
import pytest
import torch

from test_tabulate_pairs_gpu import LOWER, MAX, ROWS, S0, S1, UPPER, _poly

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [5, 2500, 7200])
@pytest.mark.parametrize("M", [1, 31, 32, 33, 65, 96, 97])
def test_widths(dpb, dtype, n, M):
    """Per entry within 2^-p (terms + 16) sum |terms|, p = 24 or 53, of sums of 4
    slots x 6 powers (forward, grad_grad) or M channels x 6 (gradient)."""
    eps = 2.0 ** (-24 if dtype == "float32" else -53)
    rng = np.random.default_rng(n + M)
    npt, k = np.dtype(dtype), 4
    T = rng.normal(0, 1, (ROWS, M, 6)).astype(npt).astype(np.float64)
    x = np.sort(np.round(rng.uniform(LOWER - 0.5, MAX + 0.5, (n, k)) * 1024) / 1024, 1)[:, ::-1]
    em = np.concatenate([x[..., None], rng.normal(0, 1, (n, k, 3))], -1)
    em[::3, 2:, 0], em[::3, 2:, 1:] = -0.75, 0.0  # folded rows
    em = em.astype(npt).astype(np.float64)
    dy, gx, ge = (rng.normal(0, 1, s).astype(npt).astype(np.float64)
                  for s in ((n, 4, M), (n, k), (n, k, 4)))
    w = np.ones((n, k))
    w[::3, 2], w[::3, 3:] = 2.0, 0.0
    v, g = _poly(T, em[..., 0])
    dev = lambda a: torch.tensor(a, dtype=getattr(torch, dtype), device="cuda")  # noqa: E731
    info = torch.tensor([LOWER, UPPER, MAX, S0, S1, -1.0], dtype=getattr(torch, dtype))
    table, e, ex = dev(T.reshape(ROWS, -1)), dev(em), dev(em[..., 0].copy())
    ops = torch.ops.deepmd
    out, = ops.tabulate_fusion_se_a(table, info, ex, e, M)
    dx, de = ops.tabulate_fusion_se_a_grad(table, info, ex, e, dev(dy), out)
    dz, = ops.tabulate_fusion_se_a_grad_grad(table, info, ex, e, dev(gx), dev(ge), out, True)
    av, ag = (np.abs(a) + 4 * np.abs(T).max() for a in (v, g))

    def check(got, want, mag, terms):
        err = np.abs(got.cpu().numpy().astype(np.float64).reshape(want.shape) - want)
        assert (err <= eps * (terms + 16) * (mag + 1e-30)).all(), float((err / mag).max() / eps)

    def slots(a, b):
        return np.einsum("ns,nsd,nsm->ndm", w, a, b)

    ae = np.abs(em)
    check(out, slots(em, v), slots(ae, av), 6 * k)
    check(dx, w * np.einsum("nsm,nsd,ndm->ns", g, em, dy),
          w * np.einsum("nsm,nsd,ndm->ns", ag, ae, np.abs(dy)), 6 * M)
    check(de, w[..., None] * np.einsum("nsm,ndm->nsd", v, dy),
          w[..., None] * np.einsum("nsm,ndm->nsd", av, np.abs(dy)), 6 * M)
    check(dz, slots(ge, v) + slots(gx[..., None] * em, g),
          slots(np.abs(ge), av) + slots(np.abs(gx)[..., None] * ae, ag), 12 * k)
