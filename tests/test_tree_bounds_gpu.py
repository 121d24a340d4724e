"""Keys out of order, which only an expired wait of the radix sort could hand to
the tree: the build ends, stays in bounds and counts what it drops, the walks
over such a tree end and report it, and the handle goes on to build correct
trees."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


def _probe(b, xm, keys):
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    dt = np.int32 if b.key_bits == 10 else np.int64
    k = torch.tensor(keys.astype(np.uint64).astype(dt), device=xm.device)
    order = torch.arange(keys.size, dtype=torch.int32, device=xm.device)
    lib_mod.call("gb_bh_tree_probe", b.handle, xm.data_ptr(), k.data_ptr(), order.data_ptr(), keys.size,
                 torch.cuda.current_stream(xm.device).cuda_stream)
    torch.cuda.synchronize()


def _disk(dev, n, seed):
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, _, mass = ic.exponential_disk(n, seed=seed)
    return torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=dev)


def _out_of_order(kind, n, bits):
    i = np.arange(n)
    if kind == "random":
        return np.random.default_rng(n).integers(0, 1 << 3 * bits, n)
    return i % (2 if kind == "alternating" else 3) << 3 * bits - 2  # 512, 342 subtrees left of a unit


@pytest.mark.parametrize("bits", [10, 21])
@pytest.mark.parametrize("n", [2, 512, 513, 3000, 20000, 100000])
@pytest.mark.parametrize("kind", ["random", "alternating", "period 3"])
def test_tree_over_keys_out_of_order(cuda_dev, n, bits, kind):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    xm = _disk(cuda_dev, n, 1)
    b = bhmod.BarnesHut(n, theta=0.5, softening=0.05, key_bits=bits, device=cuda_dev)
    _probe(b, xm, _out_of_order(kind, n, bits))
    bad = b.diag(reset=True)["bad_tree"]
    # Over two units and more something is dropped; one unit joins all its leaves.
    assert (bad > 0) == (n >= 3000)
    ref = bhmod.BarnesHut(n, theta=0.5, softening=0.05, key_bits=bits, device=cuda_dev)
    b.build(xm)
    ref.build(xm)
    got, want = b.tree_arrays(), ref.tree_arrays()
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    assert b.diag()["bad_tree"] == 0
    b.close()
    ref.close()


@pytest.mark.parametrize("n,bits", [(2, 21), (513, 10), (20000, 21), (100000, 10)])
def test_tree_over_sorted_keys_is_that_of_the_build(cuda_dev, n, bits):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    xm = _disk(cuda_dev, n, 2)
    ref = bhmod.BarnesHut(n, theta=0.5, softening=0.05, key_bits=bits, device=cuda_dev)
    ref.build(xm)
    want = ref.tree_arrays()
    b = bhmod.BarnesHut(n, theta=0.5, softening=0.05, key_bits=bits, device=cuda_dev)
    b.build(xm.flip(0).contiguous())
    _probe(b, xm[torch.tensor(want["order"].astype(np.int64), device=cuda_dev)].contiguous(), want["code"])
    got = b.tree_arrays()
    for k in want:
        if k != "order":  # the particles came in key order
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    assert b.diag()["bad_tree"] == 0
    b.close()
    ref.close()


def test_probe_checks_its_arguments(cuda_dev):
    pkg = importlib.import_module(PKG_NAME)
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    xm = _disk(cuda_dev, 10, 3)
    b = bhmod.BarnesHut(10, theta=0.5, softening=0.05, device=cuda_dev)
    for h, x, k, n in ((None, xm, xm, 10), (b.handle, None, xm, 10), (b.handle, xm, None, 10), (b.handle, xm, xm, 0),
                       (b.handle, xm, xm, 11)):
        ptrs = [None if t is None else t.data_ptr() for t in (x, k)]
        with pytest.raises(pkg.GravityError) as e:
            lib_mod.call("gb_bh_tree_probe", h, *ptrs, xm.data_ptr(), n, None)
        assert e.value.status == lib_mod.GB_EINVAL
    b.close()


@pytest.mark.parametrize("n,shape,theta", [(3000, -1, 0.5), (10000, -1, 0.5), (30000, -1, 0.5), (70000, -1, 0.5),
                                           (3000, 3, 0.5), (30000, -1, 1.3), (140000, -1, 1.0)])
@pytest.mark.parametrize("kind", ["random", "alternating"])
def test_walk_over_an_inconsistent_tree(cuda_dev, n, shape, theta, kind):
    """The nodes that were not made keep the records of the build before, of a
    larger system: their children lie past this one's nodes, or form cycles.
    Sizes: every group width of the walk in rounds (4, 8, 16 and 32 targets), the
    group walk, and the walks per lane and per warp."""
    pkg = importlib.import_module(PKG_NAME)
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    big, xm = _disk(cuda_dev, 2 * n, 4), _disk(cuda_dev, n, 5)
    b = bhmod.BarnesHut(2 * n, theta=theta, softening=0.05, max_stack=1 << 20, device=cuda_dev, check=True)
    b.set_traversal(shape)
    b.build(big)
    _probe(b, xm, _out_of_order(kind, n, 21))
    for phi in (None, torch.zeros(n, dtype=torch.float32, device=cuda_dev)):
        acc = torch.zeros_like(xm)
        b.diag(reset=True)  # the build's own count
        with pytest.raises(pkg.GravityError, match="inconsistent tree") as e:
            b.accel(acc, phi=phi)
        assert e.value.status == lib_mod.GB_EINVAL
    out, want = torch.zeros_like(big), torch.zeros_like(big)
    b.compute(big, out)  # a checked call: raises if it counts anything
    ref = bhmod.BarnesHut(2 * n, theta=theta, softening=0.05, max_stack=1 << 20, device=cuda_dev, check=True)
    ref.set_traversal(shape)
    ref.compute(big, want)
    assert torch.equal(out, want)
    b.close()
    ref.close()
