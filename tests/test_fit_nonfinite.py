"""Weights with NaN or infinity make an evaluator whose results are NaN, as plain
arithmetic does; they are no error."""

import importlib

import numpy as np
import pytest


def _params(bad):
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    p = wl.init_params(wl.SeAConfig(), seed=3)
    for f in p.fit:
        layers = [(W.copy(), b, None if d is None else d.copy()) for W, b, d in f["layers"]]
        if bad == "idt":
            layers[2][2][7] = np.inf
        else:
            layers[1][0][5, 7] = layers[2][0][3, 2] = bad
        f["layers"] = layers
    return p


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, "idt"])
def test_operand_scales(dpb, bad):
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    for v in model._FittingTC._operand_scales(_params(bad)).values():
        assert np.isfinite(v).all() and (v > 0).all()
        assert (np.frexp(v)[0] == 0.5).all()  # powers of two


def test_operand_scales_cover_their_bounds(dpb):
    """Finite weights: the bound times the scale stays in (2^11, 2^13]."""
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    p = wl.init_params(wl.SeAConfig(), seed=4)
    sc = model._FittingTC._operand_scales(p)
    for t, f in enumerate(p.fit):
        (_, _, _), (_, _, d2), (_, _, d3) = f["layers"]
        g3 = float((np.abs(f["out"][0][:, 0]) * np.abs(d3)).max())
        for v, b in ((sc["H1"][t], 1.0), (sc["H2"][t], 1 + float(np.abs(d2).max())),
                     (sc["G3"][t], g3)):
            assert 2.0 ** 11 < v * b <= 2.0 ** 13


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, "idt"])
def test_evaluator_returns_nan(dpb, bad):
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    coord, atype, box = wl.water_frame(3, seed=1)
    p = model.prepare(_params(bad), coord, atype, box)
    e, f, _ = model.SeAEvaluator(p, atype, box).compute(coord)
    assert np.isnan(e) and np.isnan(f).any()
