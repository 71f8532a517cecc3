"""The builds at the sizes where their tiles, panels and blocks end, against plain torch (B200)."""

from __future__ import annotations

import numpy as np
import pytest

from hafnium_b200.basis import ShellTable
from hafnium_b200.jk import B200DensityFittedCoulombExchange
from hafnium_b200.molecule import water_cluster
from tests.test_gpu_coulomb import hydrogens

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


# blocks of 64: one, a ragged one, several, with and without a remainder
@pytest.mark.parametrize("n_aux", [1, 63, 64, 65, 127, 128, 130, 193, 256, 257, 321, 450])
def test_the_fit_at_the_factors_block_edges(n_aux):
    import torch

    two_body = hydrogens(20, n_aux)
    eye = torch.eye(20, dtype=torch.float64, device="cuda")
    b = two_body.orbital_tensor(eye, eye).reshape(n_aux, -1)
    metric = torch.as_tensor(two_body.context.metric()).cuda()
    three = torch.as_tensor(two_body.context.three_center()).cuda().reshape(n_aux, -1)
    low = torch.linalg.cholesky(metric)
    expected = torch.linalg.solve_triangular(low, three, upper=False)  # one shell per function: the same order
    condition = float(torch.linalg.cond(metric))
    bound = 8 * n_aux * EPS * condition * float(expected.abs().max())
    assert float((b - expected).abs().max()) < bound
