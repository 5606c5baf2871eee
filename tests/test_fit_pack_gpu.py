"""The fitting weights are packed when the object is made: its first step can be
captured, or run on another stream."""

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split_b", [0, 1])
def test_first_step_under_capture(dpb, split_b):
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    at = importlib.import_module("deepmd_kit_lr_pt_b200.autotune")
    p = model.init_params(model.SeAConfig(), seed=6)
    n = 200
    D = torch.tensor(np.random.default_rng(6).normal(size=(n, 1600)).astype(np.float32) * 0.05,
                     device="cuda")
    scale = torch.full((n,), 2.0 ** 13, device="cuda")
    at.set_knob("fit_split_b", split_b)
    try:
        ref = model._FittingTC(p, [80, 120], "cuda")
        want = torch.zeros_like(D)
        ref.layers(D, want, row_scale=scale)
        fit = model._FittingTC(p, [80, 120], "cuda")
        got = torch.zeros_like(D)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            fit.layers(D, got, row_scale=scale)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        at.set_knob("fit_split_b", 0)
    assert torch.equal(got, want) and bool(got.any())


@pytest.mark.parametrize("fused", [True, False])
def test_batch_keeps_one_form(dpb, fused):
    """The batched step on Chebyshev nets holds no TF32 weights beside the FP16
    pairs it runs on."""
    wl = importlib.import_module("deepmd_kit_lr_pt_b200.workload")
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    batch = importlib.import_module("deepmd_kit_lr_pt_b200.batch")
    coord, atype, box = wl.water_frame(3, seed=2)
    p = model.prepare(model.init_params(model.SeAConfig(), seed=2), coord, atype, box)
    ev = batch.BatchEvaluator(p, [(coord, atype, box)], fused=fused)
    e, f, _ = ev.compute()
    assert ev.ptab.nets is not None and not ev.fit._tf32 and len(ev.fit._f16) == 6
    assert np.isfinite(e).all() and np.abs(f).max() > 0
