"""Small sorts (blocks of 1,024 keys sorted in shared memory, then ranked
against each other): keys and order against numpy's stable argsort at the
edges of blocks, of the ranking's stages (4 blocks) and of its CTAs (256 keys),
and at the change to one kernel per digit."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [21, 10])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 1023, 1024, 1025, 2047, 4096, 4097, 17000, 32769, 49152, 49153,
                               98304, 98305, 131072, 131073, 262144, 262145])
def test_small_sort(cuda_dev, orc, n, bits):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3)).astype(np.float32).astype(np.float64)
    if n > 100:
        pos[rng.integers(0, n, n // 3)] = pos[7]  # a third of the keys equal
    mass = np.full(n, 1.0 / n)
    b = bhmod.BarnesHut(n, theta=0.5, softening=0.05, key_bits=bits, device=cuda_dev)
    b.build(torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=cuda_dev))
    codes = orc.morton_codes(pos, bits)
    order = np.argsort(codes, kind="stable")
    np.testing.assert_array_equal(b.export("order"), order)
    np.testing.assert_array_equal(b.export("code"), codes[order])
    assert b.diag()["bad_tree"] == 0
    b.close()
