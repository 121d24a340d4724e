"""The second level of the radix sort's look-back, over groups of 16 tiles: its
waits are bounded too, and both ways of finding a group's sum give the prefix."""
import ctypes
import importlib

import pytest
import torch

from conftest import PKG_NAME


def _probe(publish, limit=1000):
    lib = importlib.import_module(PKG_NAME + "._lib").load()
    excl, timeouts = (ctypes.c_uint32 * 256)(), ctypes.c_uint64(7)
    return lib.gb_sort_group_wait_probe(limit, publish, excl, ctypes.byref(timeouts)), list(excl), timeouts.value


@pytest.mark.gpu
def test_group_waits_time_out_and_report(cuda_dev):
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    rc, _, timeouts = _probe(0)
    assert rc == lib_mod.GB_ETIMEOUT and timeouts == 256
    x = torch.arange(8, dtype=torch.float32, device=cuda_dev)  # the context still works
    assert float((x * 2).sum()) == 56.0


@pytest.mark.gpu
@pytest.mark.parametrize("publish", [1, 2])
def test_group_prefixes(cuda_dev, publish):
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    rc, excl, timeouts = _probe(publish)
    assert rc == lib_mod.GB_OK and timeouts == 0
    assert excl == [16 * d for d in range(256)]


def test_group_probe_rejects_bad_arguments_without_gpu(pkg):
    lib_mod = importlib.import_module(PKG_NAME + "._lib")
    for publish, limit in ((-1, 10), (3, 10), (0, 0), (1, (1 << 20) + 1)):
        assert _probe(publish, limit)[0] == lib_mod.GB_EINVAL
    assert lib_mod.load().gb_sort_group_wait_probe(10, 0, None, None) == lib_mod.GB_EINVAL
