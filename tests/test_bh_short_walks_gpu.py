"""The walks that expand one node at a time, at the opening angles from which they
run: against the FP64 oracle (tolerances of the other traversal tests: median <=
1e-5, 99th percentile <= 1e-4, max <= 1e-2), and against the walk in rounds at
the next smaller opening angle.  The two angles differ in their last bit, which
decides an acceptance test in about one of 10^7: at least 99.9% of the particles
get the same bits."""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu

# Particles and the opening angle of the change: per lane up to 131,071, per warp above.
LINES = [(12000, 1.4), (25000, 1.3), (39999, 1.3), (40000, 1.2), (50000, 1.1), (85001, 1.0), (131071, 1.0), (131072, 1.0),
         (150001, 0.95), (300000, 0.9), (500001, 0.85), (1200000, 0.8)]


def _case(n, seed, kind):
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, vel, mass = getattr(ic, kind)(n, seed=seed)
    return [np.asarray(a, np.float32).astype(np.float64) for a in (pos, vel, mass)]


def _records(dev, a, b):
    return torch.tensor(np.column_stack((a, b)), dtype=torch.float32, device=dev)


def _solver(dev, n, theta, bits=21, max_stack=64):
    bhmod = importlib.import_module(PKG_NAME + ".solvers.barnes_hut")
    return bhmod.BarnesHut(n, theta=theta, softening=0.05, key_bits=bits, max_stack=max_stack, G=1.0, device=dev)


def _below(theta):
    return float(np.nextafter(np.float32(theta), np.float32(0)))


def _same_rows(x, y):
    same = (x == y).reshape(x.shape[0], -1).all(1).float().mean()
    assert float(same) >= 0.999, float(same)


def _rel(a, ref):
    return np.linalg.norm(a - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-300)


def _check(rel):
    assert np.median(rel) < 1e-5 and np.percentile(rel, 99) < 1e-4 and rel.max() < 1e-2, rel.max()


@pytest.mark.parametrize("max_stack", [64, 8])
@pytest.mark.parametrize("n,theta", LINES)
def test_same_bits_on_both_sides_of_the_line(cuda_dev, n, theta, max_stack):
    pos, vel, mass = _case(n, n, "plummer")
    out, counts = [], []
    for th in (theta, _below(theta)):
        b = _solver(cuda_dev, n, th, max_stack=max_stack)
        xm, v4 = _records(cuda_dev, pos, mass), _records(cuda_dev, vel, np.zeros(n))
        acc, acc2, part = torch.zeros_like(xm), torch.zeros_like(xm), torch.ones_like(xm)
        phi = torch.zeros(n, device=cuda_dev)
        b.compute(xm, acc, phi=phi)
        b.accel_range(part, n // 3, n - n // 3, accumulate=True)
        b.diag(reset=True)
        b.compute(xm, acc2, count_work=True)
        counts.append(b.diag())
        step = acc.clone()
        b.kdk(xm, v4, step, 1e-3)
        out.append([acc, phi, part, step, xm, v4])
        assert torch.equal(acc, acc2)
        b.close()
    for x, y in zip(*out):
        _same_rows(x, y)
    for k in ("lane_interactions", "lane_tests", "stack_drops"):
        x, y = counts[0][k], counts[1][k]
        assert abs(x - y) <= 1e-4 * y + 2, (k, x, y)
    assert (counts[0]["stack_drops"] > 0) == (max_stack == 8)
    assert counts[0]["bad_tree"] == counts[0]["stack_overflow"] == 0


@pytest.mark.parametrize("n,theta,bits,kind", [(25001, 1.3, 21, "exponential_disk"), (100003, 1.0, 10, "exponential_disk"),
                                               (131072, 1.0, 21, "plummer"), (131075, 1.6, 10, "exponential_disk"),
                                               (500001, 0.85, 21, "exponential_disk")])
def test_short_walks_match_oracle(cuda_dev, orc, n, theta, bits, kind):
    pos, _, mass = _case(n, 7, kind)
    b = _solver(cuda_dev, n, theta, bits)
    xm = _records(cuda_dev, pos, mass)
    acc, phi = torch.zeros_like(xm), torch.zeros(n, device=cuda_dev)
    b.compute(xm, acc, phi=phi)
    t = orc.bh_tree(pos, mass, bits=bits)
    targets = np.random.default_rng(n).choice(n, 2000, replace=False)
    args = (pos, t["order"], t["com"], t["nmass"], t["nmin"], t["nmax"], t["left"], t["right"], theta, 0.0025)
    ref, _ = orc.traverse(*args, 1.0, targets=targets)
    ref_phi, _ = orc.traverse_phi(*args, targets=targets)
    _check(_rel(acc[:, :3].double().cpu().numpy()[targets], ref))
    _check(np.abs(phi.double().cpu().numpy()[targets] - ref_phi) / ref_phi)
    d = b.diag()
    assert d["bad_tree"] == 0 and d["stack_overflow"] == 0 and d["stack_drops"] == 0
    part, ppart = torch.zeros_like(acc), torch.zeros_like(phi)
    for s0, s1 in ((0, 1), (1, n // 3), (n // 3, n)):  # ranges cut warps: the same bits
        b.accel_range(part, s0, s1 - s0, phi=ppart)
    assert torch.equal(part, acc) and torch.equal(ppart, phi)
    b.close()
