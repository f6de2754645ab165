"""The batched launches' tile division, compiled for the host, against integer division."""
from __future__ import annotations

import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def hostdiv(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("hostdiv") / "hostdiv.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so,
                    os.path.join(ROOT, "tests", "hostcore", "hostdiv.cpp")], check=True)
    fn = ctypes.CDLL(so).check_tile_div
    fn.restype, fn.argtypes = ctypes.c_longlong, [ctypes.c_longlong] * 3
    return fn


# counts of rows of tiles and of planes, around the largest that the multiply takes and far beyond
@pytest.mark.parametrize("count", [1, 2, 63, 1000, 65534, 65535, 65536, 131071, 131072, 131073, 1 << 20, (1 << 24) + 1])
def test_tile_division_equals_integer_division(hostdiv, count):
    for d in (1, 2, 3, 5, 7, 16, 31, 32, 100, 1000, 4097, 32767, 46341, 65535, 1 << 20):
        if d * count < 1 << 31:
            assert hostdiv(d, count, 1 << 22) == 0, (d, count)


@pytest.mark.gpu
def test_batch_of_a_domain_with_very_many_rows():
    """A domain one tile wide with more rows of tiles than the multiply takes, against taller tiles."""
    import torch

    from pyocean_b200 import workloads as W
    from pyocean_b200.batch import Domain, DomainBatch
    w, got = W.zstar_box(seed=1, nx=6, ny=600001, n=1, nt=1), []
    for rows in (4, 16):
        batch = DomainBatch([Domain.from_workload(w, torch.device("cuda"))], tile_rows=rows)
        batch.domains[0].workspace.fill_(255)
        batch.step(1)
        got.append(batch.state(0).clone())
    assert torch.equal(*got)
