"""The tangent pass of the embedding nets: repeatable bits with any number of
neighbor types, and its FP32 results at the edges of the 16-row groups."""

import pytest
import torch

from test_train_dmma_gpu import EDGES, _errors, _tangent_and_gradients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,sel", [(340, (30, 40)), (340, (15, 32, 9)), (340, (15, 0, 32, 3, 9))])
def test_tangent_repeats_bit_for_bit(dpb, dtype, n, sel):
    runs = [[a.clone() for a, _ in
             _tangent_and_gradients(dpb, n, sel, 16, getattr(torch, dtype))[0]] for _ in range(5)]
    for other in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(runs[0], other))


@pytest.mark.parametrize("n,sel,ax", EDGES)
def test_embedding_tangent_fp32(dpb, n, sel, ax):
    """FP32: 2e-5 of the largest, as for the weight gradients (factors of a few
    6e-8 each, at most ten in a row, and a factor ten for cancellation)."""
    tangents, _ = _tangent_and_gradients(dpb, n, sel, ax, torch.float32)
    assert max(_errors(tangents)) <= 2e-5
