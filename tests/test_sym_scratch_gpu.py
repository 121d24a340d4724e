"""The tile-pair scratch after a larger system: a smaller one, which can need
more (smaller tiles, or more source slices per tile pair), allocates nothing,
also inside a caller's stream capture, and gives the results it gives on a
handle of its own."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu

# Sizes beside a change of the slices or the tiles.
CASES = [("acc", 36000, 35000), ("acc", 51000, 49000), ("acc", 7000, 6144), ("vjp", 10000, 8192), ("vjp", 36000, 24000)]


def _solver(dev, n):
    grav = importlib.import_module(PKG_NAME + ".solvers.gravity")
    s = grav.DirectGravity(n, dev)
    s.set_variant(2)
    return s


def _inputs(dev, n):
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, vel, mass = ic.plummer(n, seed=n)
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=dev)
    lam = [torch.tensor(np.column_stack((a, np.zeros(n))), dtype=torch.float32, device=dev) for a in (vel, pos, vel)]
    return xm, lam, torch.zeros(n, dtype=torch.float32, device=dev)


def _run(kind, s, xm, lam, lm):
    """One pass, into lam[0] (and for the adjoint into all of lam and lm)."""
    if kind == "acc":
        s.acc(xm, lam[0], 1.0, 1e-4)
        return [lam[0]]
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    lib_mod.call("gb_adjoint_step", s.handle, xm.data_ptr(), *(x.data_ptr() for x in lam), lm.data_ptr(), xm.shape[0],
                 1.0, 1e-4, 1e-3, 0, torch.cuda.current_stream(xm.device).cuda_stream)
    return [*lam, lm]


@pytest.mark.parametrize("kind,large,small", CASES)
def test_a_smaller_system_allocates_nothing(cuda_dev, kind, large, small):
    s = _solver(cuda_dev, large)
    big, little = _inputs(cuda_dev, large), _inputs(cuda_dev, small)
    _run(kind, s, *big)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(cuda_dev)[0]
    _run(kind, s, *little)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info(cuda_dev)[0] == free
    s.close()


@pytest.mark.parametrize("kind,large,small", CASES)
def test_a_smaller_system_under_capture(cuda_dev, kind, large, small):
    ref = _solver(cuda_dev, small)
    want = [x.clone() for x in _run(kind, ref, *_inputs(cuda_dev, small))]
    s = _solver(cuda_dev, large)
    _run(kind, s, *_inputs(cuda_dev, large))
    little = _inputs(cuda_dev, small)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = _run(kind, s, *little)
    g.replay()
    torch.cuda.synchronize()
    for x, y in zip(out, want):
        assert torch.equal(x, y)
    del g
    s.close()
    ref.close()
