"""dpb_gemm_f64 takes as many rows as its FP32 counterpart: up to 65,535 tiles of 128."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LIMIT = 65535 * 128


def _call(cap, C, A, B, M, N, K):
    cap.call("dpb_gemm_f64", cap.ptr(C), cap.ptr(A), cap.ptr(B), None, M, N, K, K, N, N, 0, 0, 0,
             torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("M,N", [(65535 * 64, 1), (65535 * 64 + 1, 3), (LIMIT, 1), (130, 81)])
def test_row_tiles(dpb, M, N):
    A = torch.arange(M, dtype=torch.float64, device="cuda").view(M, 1) % 1021
    B = torch.arange(1, N + 1, dtype=torch.float64, device="cuda").view(1, N)
    C = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    _call(dpb._capi, C, A, B, M, N, 1)
    assert torch.equal(C, A * B)  # products of small whole numbers


def test_more_rows_are_refused(dpb):
    one = torch.zeros(1, dtype=torch.float64, device="cuda")
    with pytest.raises(dpb._capi.DPBInvalidArgument):
        _call(dpb._capi, one, one, one, LIMIT + 1, 1, 1)
