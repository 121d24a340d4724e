"""The per-particle tree walk at the edges of its group sizes and of its
stack, against the FP64 oracle.

Tolerances are those of the other traversal tests: a node whose acceptance
test sits on the FP32/FP64 rounding boundary can flip, hence median <= 1e-5,
99th percentile <= 1e-4, max <= 1e-2 per particle.
"""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


def _case(n, seed):
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, _, mass = ic.exponential_disk(max(n, 2), seed=seed)
    return [np.asarray(a[:n], np.float32).astype(np.float64) for a in (pos, mass)]


def _solver(dev, pos, mass, theta, bits):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    n = pos.shape[0]
    b = bhmod.BarnesHut(n, theta=theta, softening=0.05, key_bits=bits, device=dev)
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=dev)
    acc, phi = torch.zeros_like(xm), torch.zeros(n, device=dev)
    b.compute(xm, acc, phi=phi)
    return b, acc, phi


def _rel(a, ref):
    return np.linalg.norm(a - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-300)


def _check(rel):
    assert np.median(rel) < 1e-5 and np.percentile(rel, 99) < 1e-4 and rel.max() < 1e-2, rel.max()


# Groups of 4, 8, 16 and 32 targets start at n = 1, 8,192, 20,480 and 65,536;
# small theta fills the list up to its reserve, where nodes are expanded one
# at a time.
@pytest.mark.parametrize("n,theta,bits", [(1, 0.5, 21), (2, 0.5, 10), (5, 0.5, 21), (31, 0.5, 10), (8191, 0.5, 21),
                                          (8192, 0.5, 10), (8197, 0.7, 21), (20479, 0.5, 10), (20480, 0.5, 21),
                                          (20491, 0.8, 10), (65535, 0.6, 21), (65536, 0.5, 10), (65537, 0.8, 21),
                                          (3001, 0.1, 21), (13001, 0.1, 10), (33001, 0.15, 21), (70001, 0.2, 10)])
def test_walk_matches_oracle(cuda_dev, orc, n, theta, bits):
    pos, mass = _case(n, 50 + n)
    b, acc, phi = _solver(cuda_dev, pos, mass, theta, bits)
    if n == 1:
        assert not acc.any() and not phi.any()
        return
    t = orc.bh_tree(pos, mass, bits=bits)
    targets = np.random.default_rng(n).choice(n, min(n, 2000), replace=False)
    args = (pos, t["order"], t["com"], t["nmass"], t["nmin"], t["nmax"], t["left"], t["right"], theta, 0.0025)
    ref, _ = orc.traverse(*args, b.G, targets=targets)
    ref_phi, _ = orc.traverse_phi(*args, targets=targets)
    _check(_rel(acc[:, :3].double().cpu().numpy()[targets], ref))
    _check(np.abs(phi.double().cpu().numpy()[targets] - ref_phi) / ref_phi)
    d = b.diag()
    assert d["bad_tree"] == 0 and d["stack_overflow"] == 0 and d["stack_drops"] == 0
    # Ranges that cut groups: the same bits.
    part, ppart = torch.zeros_like(acc), torch.zeros_like(phi)
    cuts = [0, n // 3, n // 3 + 1, min(n, (2 * n) // 3 + 2), n]
    for s0, s1 in zip(cuts[:-1], cuts[1:]):
        if s1 > s0:
            b.accel_range(part, s0, s1 - s0, phi=ppart)
    assert torch.equal(part, acc) and torch.equal(ppart, phi)
    b.close()


@pytest.mark.parametrize("n", [3, 700, 8200, 21000, 66000])
def test_walk_theta_zero_visits_every_leaf(cuda_dev, n):
    """At theta = 0 every particle tests all n - 1 internal nodes and sums the
    n - 1 other leaves, so the counters are exact."""
    pos, mass = _case(n, n)
    b, _, _ = _solver(cuda_dev, pos, mass, 0.0, 21)
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=cuda_dev)
    b.diag(reset=True)
    b.compute(xm, torch.zeros_like(xm), count_work=True)
    d = b.diag()
    assert d["lane_interactions"] == n * (n - 1) and d["lane_tests"] == n * (n - 1)
    assert d["bad_tree"] == 0 and d["stack_drops"] == 0
    b.close()
