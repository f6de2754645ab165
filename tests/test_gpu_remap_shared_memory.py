"""The side-by-side remap's shared memory: column depths whose dynamic part alone is within the default limit of 48 KB but
not with the kernel's static part."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# (n0, n1, fields); a process of their own, so that no earlier call has raised a kernel's limit
CHECK = """
import numpy as np
import pyocean_b200 as P
from oracle import oracle as O
for n0, n1, nf in ((74, 70, 1), (75, 61, 1), (73, 75, 1), (48, 26, 2), (47, 40, 2), (44, 52, 2)):
    rng = np.random.default_rng(n0)
    hs, ht = rng.uniform(0.1, 3.0, (n0, 3, 7)), rng.uniform(0.1, 3.0, (n1, 3, 7))
    f, wet = rng.normal(10.0, 2.0, (nf, n0, 3, 7)), np.ones((3, 7), bool)
    got = P.remap_columns(hs, f, ht, P.PPM_H4, wet)
    for m in range(nf):
        np.testing.assert_array_equal(got[m], O.remap_columns(hs, f[m], ht, P.PPM_H4, wet))
"""


def test_depths_between_the_dynamic_and_the_whole_limit():
    r = subprocess.run([sys.executable, "-c", CHECK], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": ROOT})
    assert r.returncode == 0, r.stderr[-2000:]


def test_two_depths_from_several_threads():
    """A launch never meets the limit of another thread's depth."""
    import threading

    import torch

    from pyocean_b200 import _lib
    dev, fn, bad = torch.device("cuda", 0), _lib.lib().pocean_remap_columns_f64, []
    go = threading.Barrier(8)

    def work(n):
        h = torch.full((n, 4, 4), 2.0, device=dev, dtype=torch.float64)
        f, w = torch.rand_like(h), torch.ones((4, 4), device=dev, dtype=torch.uint8)
        o, s = torch.empty_like(h), torch.cuda.Stream(dev)
        s.wait_stream(torch.cuda.current_stream(dev))
        go.wait()
        bad.extend(rc for rc in (fn(h.data_ptr(), f.data_ptr(), h.data_ptr(), w.data_ptr(), n, n, 4, 4, 1, 2,
                                    o.data_ptr(), s.cuda_stream) for _ in range(4000)) if rc)
        s.synchronize()
        if not torch.allclose(o, f, rtol=1e-12, atol=0.0):        # the same grid: the field, but for rounding
            bad.append(f"depth {n}: wrong values")

    threads = [threading.Thread(target=work, args=((76, 96)[i % 2],)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize(dev)
    assert not bad, (len(bad), bad[:3])
