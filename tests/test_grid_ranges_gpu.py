"""cell_start at the edges of its kernel's ranges (1,024 cells per CTA, probes
of 32 keys), against the oracle: integer outputs, so every comparison is
exact."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread", [(1, "line"), (33, "line"), (255, "line"), (256, "line"), (257, "line"), (3000, "line"),
                                      (3000, "point"), (40000, "point"), (40000, "two"), (100003, "line")])
def test_cell_start_ranges(cuda_dev, orc, n, spread):
    """Keys spread over the cells, all in one cell, or in the first and the
    last one (one CTA then holds all keys, or almost all hold none)."""
    ng = importlib.import_module(PKG_NAME + ".solvers.neighbor_grid")
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    if spread != "line":
        pos[1:] = np.float32(0.5) if spread == "point" else np.where(rng.random((n - 1, 1)) < 0.5, 0.0, 1.0)
        pos[0] = 0.0
    h = np.full(n, 1e-4, np.float32)
    grid = ng.NeighborGrid(n, device=cuda_dev)
    xm = torch.zeros((n, 4), dtype=torch.float32, device=cuda_dev)
    xm[:, :3] = torch.tensor(pos, device=cuda_dev)
    assert grid.rebuild(xm, torch.tensor(h, device=cuda_dev), None) == n
    ref = orc.grid_rebuild(pos.astype(np.float64), h.astype(np.float64), np.zeros(n, np.int32), 0.0)
    np.testing.assert_array_equal(grid.gsort.cpu().numpy(), ref["gsort"])
    np.testing.assert_array_equal(grid.cell_start.cpu().numpy(), ref["cell_start"])
    grid.close()
