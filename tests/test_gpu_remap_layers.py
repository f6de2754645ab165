"""The column remap around its layer counts, column groups and field pairs, with vanished, unreached and irregular layers,
against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import pyocean_b200 as P
from oracle import oracle as O
from pyocean_b200.batch import Domain, DomainBatch

pytestmark = pytest.mark.gpu

LAYERS = [(1, 1), (1, 3), (2, 1), (3, 3), (4, 4), (5, 7), (20, 20), (31, 33), (32, 29), (33, 65), (75, 50), (96, 96),
          (60, 96), (97, 97), (40, 97)]


def _columns(seed, n0, n1, ny, nx, nf):
    rng = np.random.default_rng(seed)
    hs, ht = rng.uniform(0.1, 3.0, (n0, ny, nx)), rng.uniform(0.1, 3.0, (n1, ny, nx))
    kind = np.arange(ny * nx).reshape(ny, nx) % 11
    hs[:, kind == 1] *= rng.random(hs[:, kind == 1].shape) > 0.4         # vanished source layers
    ht[:, kind == 2] *= rng.random(ht[:, kind == 2].shape) > 0.4         # vanished target layers
    both = kind == 3
    hs[: n0 // 2, both] = 0.0
    ht[: n1 // 2, both] = 0.0                                            # at the bottom of both
    hs[n0 // 2:, kind == 4] = 0.0                                        # at the top: few active cells
    if n0 == n1:
        ht[:, kind == 5] = hs[:, kind == 5]                              # the same grid
    tot = hs.sum(0)
    fit = kind >= 6
    scale = np.where(ht.sum(0) > 0, tot / np.where(ht.sum(0) > 0, ht.sum(0), 1.0), 1.0)
    ht[:, fit] *= scale[fit]
    hs[:, kind == 7] = 0.0                                               # no active source cell
    ht[n1 // 2, kind == 8] = -0.5                                        # outside the sweep: the array formulation
    ht[0, kind == 9] = np.nan
    ht[-1, kind == 10] = 0.0                                             # the last target vanished
    f = rng.normal(10.0, 2.0, (nf, n0, ny, nx))
    f[..., 0] = np.round(f[..., 0])                                      # equal neighbours: flat cells
    wet = rng.random((ny, nx)) > 0.1
    wet.flat[0] = True
    return hs, f, ht, wet


@pytest.mark.parametrize("scheme", [P.PCM, P.PLM, P.PPM_H4])
@pytest.mark.parametrize("n0,n1", LAYERS)
def test_columns_around_the_layer_counts(n0, n1, scheme):
    for ny, nx, nf in ((1, 1, 1), (3, 3, 2), (5, 23, 3)):
        hs, f, ht, wet = _columns(n0 * 100 + n1 + nx, n0, n1, ny, nx, nf)
        got = P.remap_columns(hs, f, ht, scheme, wet)
        for m in range(nf):
            np.testing.assert_array_equal(got[m], O.remap_columns(hs, f[m], ht, scheme, wet))


@pytest.mark.parametrize("scale", [1e-280, 1e-130, 1e-20, 1e130, 1e280])
def test_thicknesses_outside_the_short_quotients(scale):
    hs, f, ht, wet = _columns(3, 24, 24, 4, 22, 2)
    with np.errstate(all="ignore"):
        got = P.remap_columns(hs * scale, f, ht * scale, P.PPM_H4, wet)
        for m in range(2):
            np.testing.assert_array_equal(got[m], O.remap_columns(hs * scale, f[m], ht * scale, P.PPM_H4, wet))


@pytest.mark.parametrize("nf_mode", [1, 2])
@pytest.mark.parametrize("deep", [75, 100])
def test_batched_columns_of_different_depths(nf_mode, deep):
    """A batch remaps each domain as the domain alone (``deep`` above and below the layer limit of the parallel form)."""
    import torch

    from pyocean_b200 import workloads as W
    ws = [W.zstar_box(seed=s, nx=nx, ny=ny, n=n, nt=nt) for s, (nx, ny, n, nt) in
          enumerate([(21, 13, deep, 1), (9, 30, 30, 3), (33, 8, 17, 2)])]
    doms = [Domain.from_workload(w, torch.device("cuda")) for w in ws]
    batch = DomainBatch(doms, remap_nf=nf_mode)
    batch.step(1)
    for i, w in enumerate(ws):
        adv = P.TracerAdvection(scheme="weno5", time="ssprk3", dt=w.dt)
        adv.per = P.Periodic(w.periodic)
        ref = P.remap_columns(w.h_src, adv.advect_fct(w.C, w.V0, w.V1, w.Qx, w.Qy, w.ok), w.h_tgt, w.remap_scheme, w.wet)
        np.testing.assert_array_equal(batch.state(i).cpu().numpy(), ref)


def test_deep_pairs_of_a_large_plane():
    """Deep field pairs of a plane that fills the chip go by the sweep, single fields layer by layer: same values."""
    import torch
    hs, f, ht, wet = (torch.from_numpy(x).cuda() for x in _columns(17, 75, 75, 388, 389, 3))
    got = P.remap_columns(hs, f, ht, P.PPM_H4, wet)
    for m in range(3):
        one = P.remap_columns(hs, f[m:m + 1].contiguous(), ht, P.PPM_H4, wet)
        assert torch.equal(got[m].view(torch.int64), one[0].view(torch.int64))
