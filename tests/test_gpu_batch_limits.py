"""Batches at the edges of their launch rules: large batches of one tracer (limited in one marching pass) and batches of
more domains than one launch's arguments hold.  Every domain's result equals the single-domain entry points', bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from pyocean_b200 import workloads as W
from pyocean_b200.batch import Domain, DomainBatch
from pyocean_b200.step import ALETracerStep

pytestmark = pytest.mark.gpu

# (nx, ny, n): cells of a strip and rows of a segment of the marching pass are 28 and 16, its CTAs' segments 64
SMALL = [(28, 64, 2), (29, 65, 1), (27, 63, 3), (57, 15, 2), (30, 17, 1), (5, 4, 2), (3, 130, 2)]


def _domain(dev, kind: str, nx: int, ny: int, n: int, nt: int, seed: int) -> Domain:
    w = W.basin(seed=seed, nx=nx, ny=ny, n=n, nt=nt) if kind == "basin" else \
        W.zstar_box(seed=seed, nx=nx, ny=ny, n=n, nt=nt)
    if kind == "open":
        w.periodic, w.open = (), ("west", "east", "south", "north")
    dom = Domain.from_workload(w, dev)
    if kind == "open":
        rng = np.random.default_rng(seed)
        dom.inflow = torch.from_numpy(10.0 + 10.0 * rng.uniform(size=w.C.shape)).to(dev)
    return dom


def _batch(name: str, dev) -> list[Domain]:
    kinds = ("box", "open", "basin")
    small = [_domain(dev, kinds[i % 2], *s, 1, 60 + i) for i, s in enumerate(SMALL)]
    if name == "many":                                   # 3 launches; the middle one mixes tracer counts
        return [_domain(dev, kinds[i % 2], 5 + i % 9, 4 + i % 7, 1 + i % 3, 2 if i == 80 else 1, i) for i in range(130)]
    large = [_domain(dev, "basin", 230, 200, 24, 1, 7), _domain(dev, "open", 200, 129, 30, 1, 8),
             _domain(dev, "box", 141, 100, 20, 1, 9)]
    return large + small


@pytest.mark.parametrize("name,mixed", [("large", False), ("large", True), ("many", False)])
def test_batch_equals_each_domain_alone(name, mixed):
    dev = torch.device("cuda", 0)
    batch = DomainBatch(_batch(name, dev), mixed=mixed)
    if name == "large":
        assert sum(d.shape[1] * d.shape[2] * d.shape[3] for d in batch.domains) >= 1 << 21
    batch.step(2)
    torch.cuda.synchronize()
    for i, dom in enumerate(_batch(name, dev)):
        nt, n, ny, nx = dom.shape
        st = ALETracerStep(nt, n, ny, nx, dom.dt, dom.flags, dom.remap_scheme, device=dev, mixed=mixed)
        c, nxt = dom.C.clone(), torch.empty_like(dom.C)
        for _ in range(2):
            a = st.advect(c, dom.V0, dom.V1, dom.Qx, dom.Qy, dom.ok, inflow=dom.inflow)
            st.remap(dom.h_src, a, dom.h_tgt, dom.wet, nxt)
            c, nxt = nxt, c
        assert torch.equal(batch.state(i), c), f"domain {i} {dom.shape}"
