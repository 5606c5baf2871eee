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
