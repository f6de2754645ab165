"""Planes of columns with negative or NaN target thicknesses, side by side with regular ones, against the oracle bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest

import pyocean_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _columns(seed, n0, n1, ny, nx, nf):
    rng = np.random.default_rng(seed)
    hs, ht = rng.uniform(0.1, 3.0, (n0, ny, nx)), rng.uniform(0.1, 3.0, (n1, ny, nx))
    ht *= hs.sum(0) / ht.sum(0)
    kind = np.arange(ny * nx).reshape(ny, nx) % 13
    put = lambda k, a, v: a.__setitem__((rng.integers(0, a.shape[0]), kind == k), v)      # noqa: E731
    put(0, ht, -0.5)
    put(1, ht, np.nan)
    put(2, ht, -1e3)                                          # back beyond the bed
    for _ in range(4):
        put(3, ht, -rng.uniform(0.0, 2.0))
    ht[:, kind == 4] *= -1.0
    put(5, ht, -0.1)
    ht[:, kind == 5] *= rng.random(ht[:, kind == 5].shape) > 0.4          # vanished targets too
    put(6, ht, -0.1)
    hs[:, kind == 6] *= rng.random(hs[:, kind == 6].shape) > 0.4          # vanished and negative source layers
    put(6, hs, -0.2)
    put(7, ht, -0.1)
    put(7, hs, np.nan)
    put(8, ht, -0.1)
    hs[:, kind == 8] = 0.0                                    # no active source cell
    put(9, ht, np.inf)
    put(9, ht, -np.inf)
    put(10, ht, -0.0)
    put(11, hs, np.inf)
    put(11, ht, -0.3)                                         # 12: regular
    f = rng.normal(10.0, 2.0, (nf, n0, ny, nx))
    wet = rng.random((ny, nx)) > 0.1
    return hs, f, ht, wet


@pytest.mark.parametrize("scheme", [P.PCM, P.PLM, P.PPM_H4])
@pytest.mark.parametrize("n0,n1", [(1, 1), (1, 5), (3, 2), (4, 4), (20, 20), (31, 50), (50, 31), (75, 75), (96, 96), (97, 60)])
def test_irregular_columns(n0, n1, scheme):
    for ny, nx, nf in ((3, 13, 1), (4, 41, 3)):
        hs, f, ht, wet = _columns(n0 + 7 * n1 + nx, n0, n1, ny, nx, nf)
        with np.errstate(all="ignore"):
            got = P.remap_columns(hs, f, ht, scheme, wet)
            for m in range(nf):
                np.testing.assert_array_equal(got[m], O.remap_columns(hs, f[m], ht, scheme, wet))


@pytest.mark.parametrize("n,ny,nx,nf", [(20, 150, 167, 2), (20, 150, 166, 2), (50, 143, 141, 1), (75, 60, 75, 3), (96, 105, 100, 1)])
def test_around_the_launch_of_their_own(n, ny, nx, nf):
    hs, f, ht, wet = _columns(n, n, n, ny, nx, nf)
    with np.errstate(all="ignore"):
        got = P.remap_columns(hs, f, ht, P.PPM_H4, wet)
        for m in range(nf):
            np.testing.assert_array_equal(got[m], O.remap_columns(hs, f[m], ht, P.PPM_H4, wet))


@pytest.mark.parametrize("side", [40, 110])
def test_batched_irregular_columns(side):
    import torch

    from pyocean_b200 import workloads as W
    from pyocean_b200.batch import Domain, DomainBatch
    ws = [W.zstar_box(seed=s, nx=side + 3 * s, ny=side - s, n=40 + s, nt=1 + s) for s in range(2)]
    doms = []
    for i, w in enumerate(ws):
        hs, _, ht, _ = _columns(i, w.h_src.shape[0], w.h_tgt.shape[0], *w.wet.shape, 1)
        w.h_src, w.h_tgt = hs, ht
        doms.append(Domain.from_workload(w, torch.device("cuda")))
    batch = DomainBatch(doms)
    batch.step(1)
    for i, w in enumerate(ws):
        adv = P.TracerAdvection(scheme="weno5", time="ssprk3", dt=w.dt)
        adv.per = P.Periodic(w.periodic)
        c = adv.advect_fct(w.C, w.V0, w.V1, w.Qx, w.Qy, w.ok)
        got = batch.state(i).cpu().numpy()
        with np.errstate(all="ignore"):
            for m in range(c.shape[0]):
                np.testing.assert_array_equal(got[m], O.remap_columns(w.h_src, c[m], w.h_tgt, w.remap_scheme, w.wet))


# planes that go by the sweep, side by side, or the pairs one way and the odd field the other
@pytest.mark.parametrize("n,ny,nx,nf", [(1, 150, 140, 1), (2, 150, 150, 3), (3, 200, 200, 3), (10, 300, 310, 3), (30, 300, 310, 3),
                                        (12, 362, 363, 3), (75, 262, 262, 3), (75, 240, 240, 3)])
def test_around_the_sweep(n, ny, nx, nf):
    hs, f, ht, wet = _columns(n, n, n, ny, nx, nf)
    with np.errstate(all="ignore"):
        got = P.remap_columns(hs, f, ht, P.PPM_H4, wet)
        for m in range(nf):
            np.testing.assert_array_equal(got[m], O.remap_columns(hs, f[m], ht, P.PPM_H4, wet))
