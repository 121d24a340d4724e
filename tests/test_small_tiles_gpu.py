"""Tile edges of the symmetric pairwise passes of small systems (tiles of 256
particles) and the sizes around the change to tiles of 512.

Tolerances are those of the other tests of the same passes: per-particle
relative error 1e-5 against the FP64 oracle for forces (every sum has at most
a few thousand FP32 terms with compensated slot sums); positions and
velocities after a few KDK steps 2e-5 and 1e-4 of the largest component.
"""
import importlib

import numpy as np
import pytest
import torch

from conftest import PKG_NAME

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _f32(a):
    return np.asarray(a, np.float64).astype(np.float32).astype(np.float64)


def _rel(a, ref):
    return np.linalg.norm(a - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-300)


@pytest.mark.parametrize("n", [255, 256, 257, 6143, 6144, 6145])
def test_direct_small_tiles_match_oracle(cuda_dev, orc, n):
    """Force, its accumulating form and the fused KDK at tile edges; the
    512-particle tiles (a band budget too small for the slots of the small
    ones) give the same force up to rounding order."""
    grav = importlib.import_module(PKG_NAME + ".solvers.gravity")
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, vel, mass = (_f32(a) for a in ic.plummer(n, seed=n))
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=cuda_dev)
    v4 = torch.zeros_like(xm)
    v4[:, :3] = torch.tensor(vel, dtype=torch.float32, device=cuda_dev)
    ref = orc.direct_acc(pos, mass, 1.0, 1e-4)
    out = []
    for band in (1 << 30, 40960):  # the smallest budget: two tile pairs of 256
        s = grav.DirectGravity(n, cuda_dev)
        s.set_tiles(2, 4, 0, 2)
        s.set_sym_band(band)
        acc = torch.full_like(xm, 7.0)
        s.acc(xm, acc, 1.0, 1e-4)
        assert _rel(acc[:, :3].double().cpu().numpy(), ref).max() < TOL
        out.append(acc[:, :3].double().cpu().numpy())
        s.acc(xm, acc, 1.0, 1e-4, accumulate=True)
        assert _rel(acc[:, :3].double().cpu().numpy(), 2.0 * ref).max() < TOL
        x1, v1, a1 = xm.clone(), v4.clone(), torch.zeros_like(xm)
        s.acc(x1, a1, 1.0, 1e-4)
        s.kdk(x1, v1, a1, 1.0, 1e-4, 1e-3, 3)
        p, v, _ = orc.kdk_direct(pos, vel, ref, mass, 1.0, 1e-4, 1e-3, 3)
        assert np.abs(x1[:, :3].double().cpu().numpy() - p).max() < 2e-5 * np.abs(p).max()
        assert np.abs(v1[:, :3].double().cpu().numpy() - v).max() < 1e-4 * np.abs(v).max()
        s.close()
    assert _rel(out[1], out[0]).max() < TOL


@pytest.mark.parametrize("n", [36001, 50001, 65536])
def test_direct_slices_match_oracle(cuda_dev, orc, n):
    """8, 4 and 2 source slices per tile pair of 512."""
    grav = importlib.import_module(PKG_NAME + ".solvers.gravity")
    ic = importlib.import_module(PKG_NAME + ".ic")
    pos, _, mass = (_f32(a) for a in ic.plummer(n, seed=n))
    xm = torch.tensor(np.column_stack((pos, mass)), dtype=torch.float32, device=cuda_dev)
    s = grav.DirectGravity(n, cuda_dev)
    s.set_variant(2)
    acc = torch.full_like(xm, 7.0)
    s.acc(xm, acc, 1.0, 1e-4)
    targets = np.random.default_rng(n).choice(n, 1024, replace=False)
    ref = orc.direct_acc(pos, mass, 1.0, 1e-4, targets)
    assert _rel(acc[:, :3].double().cpu().numpy()[targets], ref).max() < TOL
    s.close()


@pytest.mark.parametrize("prime", [0, 1])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 8191, 8192, 8193])
def test_adjoint_small_tiles_match_large_tiles(cuda_dev, n, prime):
    """One backward step in small tiles against the same step in tiles of 512
    (what the smallest band budget selects): same inputs, FP32 summation order
    the only difference.  The per-target form is no reference here: it leaves
    the rounding of each particle's self pair, which the tiles skip."""
    grav = importlib.import_module(PKG_NAME + ".solvers.gravity")
    ic = importlib.import_module(PKG_NAME + ".ic")
    lib = importlib.import_module(PKG_NAME + "._lib")
    p, _, m = ic.exponential_disk(max(n, 2), total_mass=5.0, seed=n)
    xm = torch.zeros((n, 4), dtype=torch.float32, device=cuda_dev)
    xm[:, :3] = torch.tensor(p[:n], device=cuda_dev)
    xm[:, 3] = torch.tensor(m[:n], device=cuda_dev)
    gen = torch.Generator().manual_seed(n)
    base = [torch.randn((n, 4), generator=gen).to(cuda_dev) for _ in range(3)]
    stream = torch.cuda.current_stream(cuda_dev).cuda_stream
    out = []
    for band in (40960, 1 << 30):
        s = grav.DirectGravity(n, cuda_dev)
        s.set_sym_band(band)
        lib.call("gb_adjoint_set_variant", s.handle, 2)
        lx, lv, la = [b.clone() for b in base]
        lm = torch.zeros(n, dtype=torch.float32, device=cuda_dev)
        lib.call("gb_adjoint_step", s.handle, xm.data_ptr(), lx.data_ptr(), lv.data_ptr(), la.data_ptr(),
                 lm.data_ptr(), n, 43009.1725, 0.05 ** 2, 1e-3, prime, stream)
        out.append([t.double().cpu().numpy() for t in (lx[:, :3], lv[:, :3], la[:, :3], lm)])
        s.close()
    for a, b in zip(out[1], out[0]):
        assert np.all(np.isfinite(a))
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
