"""The descriptor passes write their per-row workspaces by row number, so a pass
over more rows than they were made for is refused on the host."""

import importlib

import numpy as np
import pytest


@pytest.mark.parametrize("layout", ["cheb", "table"])
@pytest.mark.parametrize("rows,n", [(0, 1), (8, 9), (192, 12288)])
def test_pass_over_too_many_rows_is_refused(dpb, monkeypatch, layout, rows, n):
    model = importlib.import_module("deepmd_kit_lr_pt_b200.model")
    capi = importlib.import_module("deepmd_kit_lr_pt_b200._capi")
    calls = []
    monkeypatch.setattr(model, "call", lambda *a: calls.append(a))
    monkeypatch.setattr(model, "ptr", lambda t: 0)
    tabs = object.__new__(model.PipelineTables)
    tabs.rows, tabs.nets = rows, (None if layout == "table" else object())
    tabs.info, tabs.ptrs, tabs.touched, tabs.row_scale = np.zeros(6, np.float32), None, None, None
    tabs.fwd = tabs.bwd = "f"
    sec = np.array([0, 4], np.int32)
    for one in (tabs.forward, tabs.backward):
        args = (None,) * (4 if one == tabs.forward else 5)
        with pytest.raises(capi.DPBInvalidArgument):
            one(*args, sec, n, 100, 16, 0)
        assert not calls
        one(*args, sec, rows, 100, 16, 0)
        assert calls
        calls.clear()
