"""One kernel per digit: keys and order against numpy's stable argsort at the
edges of tiles (2,048 keys) and of the look-back's groups of tiles (32,768
keys), with one handle used at several sizes in turn."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,sizes", [(10, [700001, 163839, 163840, 163841, 165889]),
                                        (21, [600000, 294911, 294912, 294913, 296961])])
def test_sort_at_tile_and_group_edges(cuda_dev, orc, bits, sizes):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    b = bhmod.BarnesHut(sizes[0], theta=0.5, softening=0.05, key_bits=bits, device=cuda_dev)
    for n in sizes:
        rng = np.random.default_rng(n)
        pos = rng.normal(size=(n, 3)).astype(np.float32).astype(np.float64)
        pos[rng.integers(0, n, n // 3)] = pos[7]  # a third of the keys equal
        xm = torch.tensor(np.column_stack((pos, np.full(n, 1.0 / n))), dtype=torch.float32, device=cuda_dev)
        b.build(xm)
        codes = orc.morton_codes(pos, bits)
        order = np.argsort(codes, kind="stable")
        np.testing.assert_array_equal(b.export("order"), order)
        np.testing.assert_array_equal(b.export("code"), codes[order])
    d = b.diag()
    assert d["bad_tree"] == 0 and d["wait_timeouts"] == 0
    b.close()
