"""prod_env_mat_a from a list whose rows hold more neighbors in range than
max_nbor_size says: up to 1,024 they are taken all the same."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("said", [1, 100, 256, 300, 512])
@pytest.mark.parametrize("n,nloc", [(480, 7), (400, 399)])
def test_rows_longer_than_said(dpb, dtype, said, n, nloc):
    cap, ops = dpb._capi, dpb.ops
    rng = np.random.default_rng(n)
    npt = np.dtype(dtype).type
    tdt = getattr(torch, dtype)
    dev = lambda a, t=None: torch.tensor(np.asarray(a), device="cuda", dtype=t)  # noqa: E731
    coord = rng.uniform(0, 4.5, (n, 3)).astype(npt)
    # every fifth center sits alone, so full and short rows share a block
    coord[2:nloc:5] += npt(1000) * np.arange(1, len(coord[2:nloc:5]) + 1, dtype=npt)[:, None]
    sec = np.array([0, 500], np.int32)
    rows = np.tile(np.arange(n, dtype=np.int32), (nloc, 1))
    rows = np.array([np.delete(r, i) for i, r in enumerate(rows)])
    avg, std = dev(np.zeros((1, 500, 4)), tdt), dev(np.ones((1, 500, 4)), tdt)
    c, t = dev(coord).view(-1), dev(np.zeros(n, np.int32))
    il, num = dev(np.arange(nloc, dtype=np.int32)), dev(np.full(nloc, n - 1, np.int32))
    rd = dev(rows)
    fn = ops._row_pointers(rd)
    sfx, s = ("f32" if dtype == "float32" else "f64"), torch.cuda.current_stream().cuda_stream

    def run(width):
        out = [torch.full((nloc, 500 * k), float("nan"), device="cuda", dtype=tdt)
               for k in (4, 12, 3)]
        nl = torch.full((nloc, 500), -7, dtype=torch.int32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        cap.call(f"dpb_prod_env_mat_a_{sfx}", *(cap.ptr(o) for o in out), cap.ptr(nl), cap.ptr(c),
                 cap.ptr(t), nloc, cap.ptr(il), cap.ptr(num), cap.ptr(fn), width, cap.ptr(avg),
                 cap.ptr(std), nloc, n, 1, ctypes.c_float(8.0), ctypes.c_float(1.0),
                 sec.ctypes.data, sec.size, cap.ptr(status), s)
        cap.call("dpb_status_check", cap.ptr(status), s)
        return [*out, nl]

    want, got = run(1024), run(said)
    assert int((want[3] >= 0).sum(1).max()) > 256
    assert all(torch.equal(a, b) for a, b in zip(want, got))
