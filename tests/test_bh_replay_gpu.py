"""One tree handle at several sizes: what a replayed step leaves on the handle
is what the same step leaves that was launched kernel by kernel on a handle of
its own.  The sizes take the sort's forms (one, two and three kernels, and one
kernel per digit), which end in buffers of their own choice only if that choice
does not depend on the size."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu

DT = 1e-4


def _state(dev, n, seed):
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, vel, mass = ic.exponential_disk(n, seed=seed)
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=dev)
    v4 = torch.tensor(np.column_stack((vel, np.zeros(n))), dtype=torch.float32, device=dev)
    return xm, v4, torch.zeros_like(xm)


def _handle(dev, n, bits, graph):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    b = bhmod.BarnesHut(n, theta=0.6, softening=0.05, key_bits=bits, device=dev)
    b.set_graph(graph)
    return b


def _left_behind(b, xm):
    """What the handle answers from its last build."""
    n = xm.shape[0]
    acc, acc_phi, part = (torch.zeros_like(xm) for _ in range(3))
    phi = torch.zeros(n, dtype=torch.float32, device=xm.device)
    b.accel(acc)
    b.accel(acc_phi, phi=phi)
    b.accel_range(part, n // 3, n - n // 3)
    return [acc, acc_phi, phi, part], b.tree_arrays()


def _assert_same(got, want, n):
    for g, w in zip(got[0], want[0]):
        assert torch.equal(g, w)
    for k in want[1]:
        np.testing.assert_array_equal(got[1][k], want[1][k], err_msg=k)
    code = got[1]["code"]
    assert np.all(code[1:] >= code[:-1]) and np.array_equal(np.sort(got[1]["order"]), np.arange(n))


@pytest.mark.parametrize("n,other,bits", [(20000, 500, 21), (500, 20000, 21), (20000, 50000, 10), (50000, 1025, 21),
                                          (300000, 10000, 21), (10000, 300000, 10)])
def test_replay_after_a_build_of_another_size(cuda_dev, n, other, bits):
    b = _handle(cuda_dev, max(n, other), bits, True)
    ref = _handle(cuda_dev, n, bits, False)
    s, s_ref, between = _state(cuda_dev, n, 1), _state(cuda_dev, n, 1), _state(cuda_dev, other, 2)
    b.kdk(*s, DT)  # captured
    b.compute(between[0], between[2])
    b.kdk(*s, DT)  # replayed
    ref.kdk(*s_ref, DT, 2)
    for x, y in zip(s, s_ref):
        assert torch.equal(x, y)
    _assert_same(_left_behind(b, s[0]), _left_behind(ref, s_ref[0]), n)
    for h in (b, ref):
        assert h.diag()["bad_tree"] == 0
        h.close()


@pytest.mark.parametrize("n,n_phi", [(500, 20000), (20000, 500), (20000, 300000)])
def test_steps_with_and_without_potential_at_two_sizes(cuda_dev, n, n_phi):
    """The two kinds of step hold a graph each; the one replayed last decides."""
    b = _handle(cuda_dev, max(n, n_phi), 21, True)
    ref, ref_phi = _handle(cuda_dev, n, 21, False), _handle(cuda_dev, n_phi, 21, False)
    s, s_ref = _state(cuda_dev, n, 3), _state(cuda_dev, n, 3)
    p, p_ref = _state(cuda_dev, n_phi, 4), _state(cuda_dev, n_phi, 4)
    phi, phi_ref = (torch.zeros(n_phi, dtype=torch.float32, device=cuda_dev) for _ in range(2))
    for _ in range(2):  # the second time both are replayed
        b.kdk(*s, DT)
        ref.kdk(*s_ref, DT)
        _assert_same(_left_behind(b, s[0]), _left_behind(ref, s_ref[0]), n)
        b.kdk(*p, DT, phi=phi)
        ref_phi.kdk(*p_ref, DT, phi=phi_ref)
        _assert_same(_left_behind(b, p[0]), _left_behind(ref_phi, p_ref[0]), n_phi)
        assert torch.equal(phi, phi_ref)
    for h in (b, ref, ref_phi):
        h.close()


@pytest.mark.parametrize("replayed", [-1, 3])
def test_groups_after_a_replay(cuda_dev, replayed):
    """The group walk after a replayed step walks that step's groups, whichever
    shape the step had and the build before it."""
    n = 20000
    b = _handle(cuda_dev, n, 21, True)
    ref = _handle(cuda_dev, n, 21, False)
    s, s_ref, between = _state(cuda_dev, n, 5), _state(cuda_dev, n, 5), _state(cuda_dev, n, 6)
    b.set_traversal(replayed)
    ref.set_traversal(replayed)
    b.kdk(*s, DT)  # captured
    b.set_traversal(2 - replayed)  # 3 and -1
    b.compute(between[0], between[2])
    b.set_traversal(replayed)
    b.kdk(*s, DT)  # replayed
    ref.kdk(*s_ref, DT, 2)
    out = []
    for h, x in ((b, s[0]), (ref, s_ref[0])):
        h.set_traversal(3)
        acc = torch.zeros_like(x)
        h.accel(acc)
        out.append(acc)
        assert h.diag()["bad_tree"] == 0
        h.close()
    assert torch.equal(s[0], s_ref[0]) and torch.equal(out[0], out[1])
