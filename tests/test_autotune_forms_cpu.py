"""The autotuner's cache tells the forms of the descriptor passes apart, and the
kernels of other builds; it tries no knob that the passes do not read."""

import importlib
import json

import pytest


@pytest.fixture()
def mods(dpb):
    return {m: importlib.import_module(f"deepmd_kit_lr_pt_b200.{m}")
            for m in ("model", "batch", "autotune")}


def _tables(model, degree, nets):
    t = object.__new__(model.PipelineTables)
    t.degree, t.nets, t.layout = degree, nets, 5 if nets is not None else degree
    return t


def _tune_calls(mods, monkeypatch, cls, **attrs):
    seen = []
    monkeypatch.setattr(mods["autotune"], "tune",
                        lambda run, cap, knobs, signature, **kw: seen.append((knobs, signature)))
    cfg = importlib.import_module("deepmd_kit_lr_pt_b200.workload").SeAConfig()
    for tab in (_tables(mods["model"], 3, object()), _tables(mods["model"], 3, None),
                _tables(mods["model"], 5, None)):
        ev = object.__new__(cls)
        ev.cfg, ev.ptab, ev.dev = cfg, tab, None
        for k, v in attrs.items():
            setattr(ev, k, v)
        ev.tune()
        ev.plan = None  # for its destructor
    return seen


def test_frame_and_batch_tune(mods, monkeypatch):
    for seen in (_tune_calls(mods, monkeypatch, mods["model"].SeAEvaluator, nloc=192,
                             mode="compressed", skin=0.0),
                 _tune_calls(mods, monkeypatch, mods["batch"].BatchEvaluator, nframes=2, N=400,
                             plan=None)):
        cheb, cubic, quintic = seen
        assert not {"desc_atoms_per_cta", "desc_coef_l1"} & set(cheb[0])
        for knobs, _ in (cubic, quintic):
            assert {"desc_atoms_per_cta", "desc_coef_l1", "fit_n_tile"} <= set(knobs)
        assert len({cheb[1], cubic[1], quintic[1]}) == 3


def test_cache_of_other_kernels_is_not_used(mods, monkeypatch, tmp_path):
    at = mods["autotune"]
    monkeypatch.setenv("DPB_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(at.torch.cuda, "get_device_name", lambda d: "gpu")
    (tmp_path / "tune.json").write_text(json.dumps({"gpu|w": {"knobs": {"fit_split_b": 1}}}))
    assert at.load_cached("w") is None
    at._store("w", None, {"knobs": {"fit_split_b": 0}})
    assert at.load_cached("w") == {"knobs": {"fit_split_b": 0}}
    monkeypatch.setattr(at, "KERNELS", at.KERNELS + 1)
    assert at.load_cached("w") is None
