"""The many-CTA solve of the reduced camera system (more than 224 unknowns) at the edges of its 64-column
blocks and of its schedules: one block row left over, a last block of two columns, tiles handed out
one and two at a time, panel CTAs taking tiles, more panel tasks than CTAs.

Against a float64 solve of the same damped system: dx is its rounding to float32 (2^-24 of its
size) on top of two FP64 solves of a system of condition below 1e7; bound 2^-23 of the largest.
"""

import numpy as np
import pytest
import torch

import droid_backends
from hislam2_b200 import backends
from test_gpu_small_solve import NAMES, window

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [38, 42, 43, 64, 75, 107, 235, 500, 800])
def test_solve_sizes(cuda, P):
    w = {k: v.to(cuda) for k, v in window(P + 1, P).items()}
    A, b = backends.ba_reduced_system(*[w[k] for k in NAMES], w["ii"], w["jj"], 1, P + 1)
    A, b = A.cpu().numpy(), b.cpu().numpy()
    A[np.diag_indices_from(A)] += 0.1 + 1e-4 * np.diagonal(A)
    x = np.linalg.solve(A, b)
    dx, _, _ = droid_backends.ba(*[w[k] for k in NAMES], w["ii"], w["jj"], 1, P + 1, 1, 1e-4, 0.1, False)
    assert np.abs(dx.cpu().numpy().reshape(-1) - x).max() <= 2 ** -23 * np.abs(x).max()


@pytest.mark.parametrize("P", [64, 235])
def test_solve_not_positive_definite(cuda, P):
    """lm = -2 makes every damped diagonal negative: dx = 0."""
    w = {k: v.to(cuda) for k, v in window(P + 1, 90).items()}
    dx, _, _ = droid_backends.ba(*[w[k] for k in NAMES], w["ii"], w["jj"], 1, P + 1, 1, -2.0, 0.0, True)
    assert torch.count_nonzero(dx) == 0
