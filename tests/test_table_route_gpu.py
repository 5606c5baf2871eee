"""Nets that do not expand in Chebyshev polynomials stay on the cubic tables: the
same frames, batches and knobs as the tests of table_degree=3 and of the
autotuner's knobs, on that route; and the table route's fitting scales."""

import importlib

import numpy as np
import pytest
import torch

import test_autotune_gpu as knobs
import test_cubic_gpu as cubic

pytestmark = pytest.mark.gpu


@pytest.fixture()
def on_tables(dpb, monkeypatch):
    table = importlib.import_module("deepmd_kit_lr_pt_b200.table")
    monkeypatch.setattr(table, "chebyshev_net", lambda *a, **k: None)
    return {m: importlib.import_module(f"deepmd_kit_lr_pt_b200.{m}")
            for m in ("model", "workload", "batch", "train", "autotune", "table", "engine")}


@pytest.fixture()
def saved_knobs(on_tables):
    at = on_tables["autotune"]
    saved = at.current()
    yield
    at.apply(saved)


def _tuple(m):
    return m["workload"], m["model"], m["table"], m["batch"]


def test_cubic_descriptor(on_tables):
    cubic.test_cubic_descriptor_matches_quintic(_tuple(on_tables))


def test_cubic_batched_and_extrapolation(on_tables):
    cubic.test_cubic_batched_and_extrapolation(_tuple(on_tables))


def test_batched_step_same_under_every_shape(on_tables, saved_knobs):
    knobs.test_batched_step_same_under_every_shape(on_tables, None)


def test_frame_step_same_under_every_shape(on_tables, saved_knobs):
    knobs.test_frame_step_same_under_every_shape(on_tables, None)


@pytest.mark.parametrize("degree", [3, 5])
def test_tensor_core_contraction(on_tables, saved_knobs, degree):
    knobs.test_tensor_core_contraction_matches(on_tables, None, degree)


@pytest.mark.parametrize("degree", [3, 5])
def test_staged_batches_agree_with_the_chebyshev_route(on_tables, monkeypatch, degree):
    """Tables against polynomials on the same frames, both with the FP16 form of
    the fitting GEMMs: energies to 1e-7, forces to 1e-6 (as degree 3 against
    degree 5)."""
    m = on_tables
    rng = np.random.default_rng(7)
    frames = [m["workload"].water_frame_density(150, rng), m["workload"].cu_frame(108, rng),
              m["workload"].water_frame_density(24, rng)]
    p = m["model"].prepare_frames(
        m["model"].init_params(m["model"].SeAConfig(sel=(46, 92, 60)), seed=2), frames)
    ev = m["batch"].BatchEvaluator(p, frames, table_degree=degree, fused=False)
    assert ev.ptab.nets is None
    E, F, V = ev.compute()
    ev.check()
    monkeypatch.undo()
    ref = m["batch"].BatchEvaluator(p, frames, fused=False)
    assert ref.ptab.nets is not None
    E0, F0, V0 = ref.compute()
    np.testing.assert_allclose(E, E0, rtol=1e-7, atol=1e-6)
    assert float(np.sqrt(np.mean((F - F0) ** 2))) < 1e-6
    np.testing.assert_allclose(V, V0, rtol=1e-6, atol=1e-5)


def test_row_scales_from_tables(on_tables):
    """Every descriptor row times its scale stays below 2^14, and above 2^8 where
    the row's bound is within 2^5 of its largest entry (few env columns)."""
    m = on_tables
    coord, atype, box = m["workload"].water_frame(4, seed=3)
    p = m["model"].prepare(m["model"].init_params(m["model"].SeAConfig(), seed=3), coord, atype,
                           box)
    ev = m["model"].SeAEvaluator(p, atype, box)
    ev.compute(coord)
    top = ev.D.abs().amax(1) * ev.ptab.row_scale
    assert float(top.max()) < 2.0 ** 14 and float(top.min()) > 2.0 ** 8
    assert bool((torch.frexp(ev.ptab.row_scale)[0] == 0.5).all())
