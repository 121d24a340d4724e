"""Adjoint segments: the last segment's positions kept from the forward pass
against the same segment re-run from its checkpoint.  The forward steps are
deterministic, so the gradients must be equal bit for bit."""
import importlib

import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu


def _gradients(adj, leaves, target, nsteps, every, passes=1):
    x, v, m = leaves
    solver = importlib.import_module(PKG_NAME + ".solvers.gravity").DirectGravity(x.shape[0], x.device)
    xt, vt = adj.simulate(x, v, m, G=43009.1725, softening=0.05, dt=1e-3, nsteps=nsteps, checkpoint_every=every,
                          solver=solver)
    loss = ((xt - target) ** 2).mean() + 1e-6 * (vt ** 2).mean()
    out = [torch.autograd.grad(loss, leaves, retain_graph=p < passes - 1) for p in range(passes)]
    solver.close()
    return out, xt.detach()


@pytest.mark.parametrize("nsteps,every", [(1, 1), (1, 5), (2, 5), (5, 5), (6, 5), (7, 5), (11, 1)])
def test_kept_segment_equals_rerun_segment(cuda_dev, monkeypatch, nsteps, every):
    adj = importlib.import_module(PKG_NAME + ".adjoint")
    ic = importlib.import_module(PKG_NAME + ".ic")
    p, v, m = ic.exponential_disk(300, total_mass=5.0 * 300 / 65536, seed=5)
    leaves = [torch.tensor(a, dtype=torch.float32, device=cuda_dev).requires_grad_(True) for a in (p, v, m)]
    target = leaves[0].detach() + 0.05
    (first, second), x1 = _gradients(adj, leaves, target, nsteps, every, passes=2)
    monkeypatch.setattr(adj, "KEEP_BYTES", 0)
    (rerun,), x2 = _gradients(adj, leaves, target, nsteps, every)
    assert torch.equal(x1, x2)
    for a, b, c in zip(first, second, rerun):
        assert torch.all(torch.isfinite(a)) and a.abs().max() > 0
        assert torch.equal(a, b) and torch.equal(a, c)
