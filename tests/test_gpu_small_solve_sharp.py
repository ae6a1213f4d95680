"""The one-CTA solve (up to 224 unknowns) held to its FP64 arithmetic: dx against a float64 solve of the
same reduced system, at every number of 16-column blocks that its range meets and on both sides of
their edges.  dx is the rounding to float32 (2^-24 of its size) of an FP64 solve of a system of
condition below 1e7; bound 2^-23 of the largest, as for the many-CTA solve.
"""

import numpy as np
import pytest
import torch

import droid_backends
from hislam2_b200 import backends
from test_gpu_small_solve import NAMES, window

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 2, 3, 5, 6, 8, 11, 13, 16, 19, 21, 24, 27, 29, 32, 35, 37])
def test_solve_sizes(cuda, P):
    w = {k: v.to(cuda) for k, v in window(P + 1, P).items()}
    A, b = backends.ba_reduced_system(*[w[k] for k in NAMES], w["ii"], w["jj"], 1, P + 1)
    A, b = A.cpu().numpy(), b.cpu().numpy()
    assert A.shape[0] == 6 * P <= 224
    A[np.diag_indices_from(A)] += 0.1 + 1e-4 * np.diagonal(A)
    x = np.linalg.solve(A, b)
    dx, _, _ = droid_backends.ba(*[w[k] for k in NAMES], w["ii"], w["jj"], 1, P + 1, 1, 1e-4, 0.1, False)
    assert np.abs(dx.cpu().numpy().reshape(-1) - x).max() <= 2 ** -23 * np.abs(x).max()
