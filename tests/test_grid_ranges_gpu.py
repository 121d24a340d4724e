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
                                      (3000, "point"), (40000, "point"), (40000, "two"), (65536, "line"), (65537, "two"),
                                      (100003, "line")])
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


@pytest.mark.parametrize("cell,offset,n", [(0.25, -3.7, 30000), (0.1, 1e3, 20000), (3e-3, 0.0, 50001), (7.3, -1e5, 10000)])
def test_cells_at_edges(cuda_dev, orc, cell, offset, n):
    """Particles on cell edges and a few ulps beside them: FP32 decides the
    cells away from edges, FP64 the others, as numpy's FP64 division does."""
    ng = importlib.import_module(PKG_NAME + ".solvers.neighbor_grid")
    rng = np.random.default_rng(n)
    edge = offset + rng.integers(0, 12, (n, 3)) * np.float64(cell)
    pos = (edge + rng.choice([0.0, 1.0], (n, 3)) * rng.normal(0.0, 1e-6 * cell, (n, 3))).astype(np.float32)
    pos += rng.integers(-2, 3, (n, 3)) * np.spacing(pos)
    h = np.full(n, 0.5 * cell, np.float32)
    star = (rng.random(n) < 0.2).astype(np.int32)
    grid = ng.NeighborGrid(n, device=cuda_dev)
    xm = torch.zeros((n, 4), dtype=torch.float32, device=cuda_dev)
    xm[:, :3] = torch.tensor(pos, device=cuda_dev)
    ngas = grid.rebuild(xm, torch.tensor(h, device=cuda_dev), torch.tensor(star, device=cuda_dev))
    ref = orc.grid_rebuild(pos.astype(np.float64), h.astype(np.float64), star, 0.0)
    assert ngas == ref["ngas"]
    np.testing.assert_array_equal(grid.gsort.cpu().numpy(), ref["gsort"])
    np.testing.assert_array_equal(grid.cell_start.cpu().numpy(), ref["cell_start"])
    grid.close()
