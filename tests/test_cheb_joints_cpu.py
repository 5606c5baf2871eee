"""The piecewise Chebyshev expansion where its intervals meet: both sides are
within the fit's bounds of the table, the left one within twice those, so the
jumps are within three times."""

import importlib

import numpy as np
import pytest


def _at(C, t, half):
    """value and slope of one interval at t"""
    k = np.arange(C.shape[0])
    T, U = [1.0, t], [1.0, 2 * t]
    for _ in range(2, C.shape[0]):
        T.append(2 * t * T[-1] - T[-2])
        U.append(2 * t * U[-1] - U[-2])
    d = np.array([0.0] + [q * U[q - 1] for q in k[1:]])
    return np.array(T) @ C, d @ C / half


@pytest.mark.parametrize("seed", range(8))
def test_jumps(dpb, seed):
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    tb = importlib.import_module("deepmd_kit_lr_pt_b200.table")
    p = wl.init_params(wl.SeAConfig(sel=(4,)), seed=seed)
    avg, std = np.tile([0.06, 0, 0, 0], (1, 4)), np.tile([0.11, 0.07, 0.07, 0.07], (1, 4))
    (table, info), = tb.build_tables(p.emb, avg, std, (4,), 0.95, 0.5, 6.0)
    C, center, half, lut = tb.chebyshev_net(table, info)
    assert (np.diff(lut.astype(int)) >= 0).all()
    first = int(round((info[1] - info[0]) / info[3]))
    rows = np.asarray(table[:first], np.float64).reshape(first, -1, 6)
    big, steep = np.abs(rows[..., 0]).max(), np.abs(rows[..., 1]).max()
    assert len(C) > 1 and np.allclose(center[:-1] + half[:-1], center[1:] - half[1:])
    for r in range(len(C)):
        for side, t in ((0, -1.0), (1, 1.0)):
            x = center[r] + t * half[r]
            k = min(int(round((x - info[0]) / info[3])), first - 1)
            u = x - (info[0] + k * info[3])
            v = sum(rows[k, :, q] * u**q for q in range(6))
            g = sum(q * rows[k, :, q] * u ** (q - 1) for q in range(1, 6))
            cv, cg = _at(C[r], t, half[r])
            # the fit's own bounds (its largest values are these or the midpoints')
            assert np.abs(cv - v).max() <= (1 + side) * 1.01 * 1.5e-8 * big
            assert np.abs(cg - g).max() <= (1 + side) * 1.01 * 5e-7 * steep
    for r in range(len(C) - 1):
        (v0, g0), (v1, g1) = _at(C[r], 1.0, half[r]), _at(C[r + 1], -1.0, half[r + 1])
        assert np.abs(v0 - v1).max() <= 3.03 * 1.5e-8 * big
        assert np.abs(g0 - g1).max() <= 3.03 * 5e-7 * steep
