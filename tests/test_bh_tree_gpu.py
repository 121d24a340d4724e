"""The tree build at the edges of its chunks (512 leaves) and of its groups of
chunks (32), and on trees whose chunks leave more subtrees than are joined at
a time, against the oracle: topology and boxes exact; FP32 node masses within
5e-6 relative and centres within 1e-5 of the system size, as in the other tree
tests."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


def _check_tree(dev, orc, pos, mass, bits):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    n = pos.shape[0]
    b = bhmod.BarnesHut(n, theta=0.5, softening=0.05, key_bits=bits, device=dev)
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=dev)
    b.build(xm)
    t = b.tree_arrays()
    codes = orc.morton_codes(pos, bits)
    order = orc.stable_argsort(codes)
    np.testing.assert_array_equal(t["order"], order)
    left, right, parent = orc.build_radix(codes[order])
    np.testing.assert_array_equal(t["left"], left)
    np.testing.assert_array_equal(t["right"], right)
    np.testing.assert_array_equal(t["parent"], parent)
    com, nmass, nmin, nmax = orc.summaries(order, pos, mass, parent)
    np.testing.assert_array_equal(t["nmin"], nmin)
    np.testing.assert_array_equal(t["nmax"], nmax)
    np.testing.assert_allclose(t["nmass"], nmass, rtol=5e-6)
    np.testing.assert_allclose(t["com"], com, rtol=0, atol=1e-5 * np.abs(pos).max())
    assert b.diag()["bad_tree"] == 0
    return b, xm


@pytest.mark.parametrize("n,bits", [(2, 21), (511, 21), (512, 10), (513, 21), (1025, 10), (16384, 21), (16385, 10),
                                    (16897, 21), (525000, 10)])
def test_tree_at_chunk_edges(cuda_dev, orc, n, bits):
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, _, mass = ic.exponential_disk(n, seed=n)
    pos, mass = [a.astype(np.float32).astype(np.float64) for a in (pos, mass)]
    if n > 600:
        pos[300:700] = pos[5]  # equal keys across chunks: the index decides
    b, _ = _check_tree(cuda_dev, orc, pos, mass, bits)
    b.close()


def _spines():
    """20 caterpillar trees of 53 bushes of 16 leaves: a bush joins only what
    follows it, so a chunk leaves about 25 subtrees and 32 chunks over 512."""
    keys = set()
    for c in range(20):
        for i in range(53):
            low = 57 - i  # bits below the spine's zero
            for leaf in range(16):
                keys.add(c << 58 | ((1 << i) - 1) << (53 - i) << 5 | leaf << max(low - 4, 0))
    keys = np.array(sorted(keys), np.int64)
    q = np.zeros((keys.size, 3), np.int64)
    for bit in range(21):
        for a in range(3):
            q[:, a] |= (keys >> (3 * bit + a) & 1) << bit
    pos = (q + 0.5) / ((2 ** 21 - 1) / 1.0000001)
    pos = np.concatenate((pos, [[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]]))
    return np.clip(pos, 0.0, 1.0).astype(np.float32).astype(np.float64)


def test_tree_with_long_spines(cuda_dev, orc):
    pos = _spines()
    rng = np.random.default_rng(3)
    mass = rng.uniform(0.5, 1.5, pos.shape[0]).astype(np.float32).astype(np.float64)
    b, _ = _check_tree(cuda_dev, orc, pos, mass, 21)
    b.close()


@pytest.mark.parametrize("n", [1, 20, 513, 20000])
def test_groups_marked_after_the_build(cuda_dev, n):
    """Selecting the group walk after a build marks its groups in a second pass:
    the same accelerations as a build in that mode."""
    ic = importlib.import_module(PKG_NAME + ".ic")
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    pos, _, mass = ic.exponential_disk(max(n, 2), seed=n)
    xm = torch.tensor(np.column_stack((pos, mass))[:n], dtype=torch.float32, device=cuda_dev)
    out = []
    for late in (False, True):
        b = bhmod.BarnesHut(n, theta=0.5, softening=0.05, device=cuda_dev)
        if not late:
            b.set_traversal(3)
        b.build(xm)
        b.set_traversal(3)
        acc = torch.full_like(xm, 7.0)
        b.accel(acc)
        out.append(acc)
        assert b.diag()["bad_tree"] == 0
        b.close()
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("extra", [0, 1])
def test_tree_at_the_change_of_block_size(cuda_dev, orc, extra):
    """One chunk per SM is the last size of the wide blocks."""
    ic = importlib.import_module(PKG_NAME + ".ic")
    n = 512 * torch.cuda.get_device_properties(cuda_dev).multi_processor_count + extra
    pos, _, mass = ic.plummer(n, seed=n)
    pos, mass = (a.astype(np.float32).astype(np.float64) for a in (pos, mass))
    b, _ = _check_tree(cuda_dev, orc, pos, mass, 21)
    b.close()
