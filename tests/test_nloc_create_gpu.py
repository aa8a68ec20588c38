"""A projector set on the device takes about the memory of its coefficients: columns
are not padded beyond an even number (the results are tested with the kernels)."""
import numpy as np
import pytest
import torch

import skgemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [2, 3, 4, 17])
def test_narrow_projectors_are_not_widened(cuda, ncol):
    K, P, nrow = 20000, 150, 4000
    rng = np.random.default_rng(ncol)
    index = np.concatenate([rng.choice(K, nrow, replace=False) for _ in range(P)])
    chi = rng.standard_normal(P * nrow * ncol)
    args = (np.full(P, nrow), np.full(P, ncol), np.arange(1, P + 1), np.arange(P + 1) * ncol,
            index, chi, rng.standard_normal(P * ncol), K)
    skgemm.NlocProjector(*args).close()  # the creation kernel's code is loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    h = skgemm.NlocProjector(*args)
    held = free - torch.cuda.mem_get_info()[0]
    rows = P * nrow
    tables = rows * (4 + 8) + 3 * K * 8
    assert held <= rows * (ncol + ncol % 2) * 8 + tables + (20 << 20)
    h.close()
