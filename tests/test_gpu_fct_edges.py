"""The FCT step's face arithmetic and passes where they can go wrong: values at the ends of the exponent range, zeros and
non-finite values through the short divisions, and grids around the tile edges, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import pyocean_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _bits_equal(a, b):
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(b)
    np.testing.assert_array_equal(np.isnan(a), nan)
    np.testing.assert_array_equal(np.where(nan, 0.0, a).view(np.int64), np.where(nan, 0.0, b).view(np.int64))


def _adv(mod, scheme, dt=1.0, per=(), open_=()):
    adv = mod.TracerAdvection(scheme=scheme, time="ssprk3", dt=dt, ob=mod.OpenEdges(open_))
    adv.per = mod.Periodic(per)
    return adv


SCALES = {"unit": 0, "tiny": -300, "subnormal": -318, "large": 150, "huge": 303}


@pytest.mark.parametrize("scheme", ["weno5", "weno5js"])
@pytest.mark.parametrize("scale", sorted(SCALES))
def test_face_values_at_the_ends_of_the_exponent_range(scheme, scale):
    rng = np.random.default_rng(SCALES[scale] + 1000)
    n, ny, nx = 2, 40, 48
    e = 10.0 ** SCALES[scale]
    with np.errstate(over="ignore"):
        c = rng.normal(0.0, 1.0, (3, n, ny, nx)) * e
    c[0] *= rng.choice([0.0, 1.0], c[0].shape)                        # zeros of both signs among the values
    c[1] = (5.0 + rng.normal(0.0, 1.0, c[1].shape) * 10.0 ** rng.integers(-16, 1, c[1].shape)) * e      # cancellation
    c[2] = e * 10.0 ** rng.uniform(-8, 4, c[2].shape)                 # neighbours many orders apart
    c[2, 0, 3::7, 2::5] = 0.0
    Qx, Qy = rng.normal(0, 1, (n, ny, nx + 1)), rng.normal(0, 1, (n, ny + 1, nx))
    Qx[:, ::5] = 0.0
    ok = rng.random((n, ny, nx)) > 0.05
    for got, ref in zip(_adv(P, scheme).faces_h(c, Qx, Qy, ok), _adv(O, scheme).faces_h(c, Qx, Qy, ok)):
        _bits_equal(got, ref)


@pytest.mark.parametrize("scheme", ["weno5", "weno5js"])
def test_face_values_of_flat_signed_zero_and_non_finite_stencils(scheme):
    rng = np.random.default_rng(5)
    n, ny, nx = 1, 24, 64
    c = np.zeros((6, n, ny, nx))
    c[0] = -0.0
    c[1] = rng.choice([0.0, -0.0], c[1].shape)
    c[2] = 17.3
    c[3] = rng.normal(size=c[3].shape)
    c[3, 0, 5, 9], c[3, 0, 11, 40], c[3, 0, 18, 21] = np.inf, -np.inf, np.nan
    c[4] = np.where(rng.random(c[4].shape) < 0.5, 1.0, 0.0)           # top-hat patches
    c[5] = rng.choice([1e154, -3e153, 1.0, 0.0, 1e-160], c[5].shape)  # squares overflow and underflow
    Qx, Qy = rng.normal(0, 1, (n, ny, nx + 1)), rng.normal(0, 1, (n, ny + 1, nx))
    ok = np.ones((n, ny, nx), bool)
    with np.errstate(all="ignore"):
        for got, ref in zip(_adv(P, scheme).faces_h(c, Qx, Qy, ok), _adv(O, scheme).faces_h(c, Qx, Qy, ok)):
            _bits_equal(got, ref)


def _domain(seed, nt, n, ny, nx, per):
    rng = np.random.default_rng(seed)
    h = rng.uniform(1.0, 3.0, (n, ny, nx))
    Qx, Qy = rng.normal(0, 0.05, (n, ny, nx + 1)), rng.normal(0, 0.05, (n, ny + 1, nx))
    if "x" in per:
        Qx[..., -1] = Qx[..., 0]
    if "y" in per:
        Qy[:, -1] = Qy[:, 0]
    V1 = h - 0.1 * (Qx[..., 1:] - Qx[..., :-1] + Qy[:, 1:] - Qy[:, :-1])
    ok = (rng.random((n, ny, nx)) > 0.1) & (V1 > 0)
    C = rng.normal(10.0, 1.0, (nt, n, ny, nx))
    if nt > 1:
        C[-1] = np.where(rng.random(C[-1].shape) < 0.5, 1.0, 0.0)
    return C, h, V1, Qx, Qy, ok


GRIDS = [(1, 1, 1, 1), (2, 1, 2, 3), (1, 3, 7, 5), (3, 2, 8, 32), (2, 2, 9, 33), (1, 2, 14, 38), (2, 1, 15, 31),
         (2, 2, 22, 69), (1, 2, 29, 61), (4, 1, 16, 96), (2, 3, 13, 101)]


@pytest.mark.parametrize("per,open_", [((), ()), (("x",), ()), (("x", "y"), ()), ((), ("west", "east", "south", "north")),
                                       (("y",), ("west",))])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_fct_step_around_the_tile_edges(grid, per, open_):
    nt, n, ny, nx = grid
    a = _domain(sum(grid) * 7, nt, n, ny, nx, per)
    infl = a[0] + 1.0 if open_ else None
    fi = nx // 2
    got, fx = _adv(P, "weno5", 0.1, per, open_).advect_fct(*a, inflow=infl, flux_face_i=fi)
    ref, rx = _adv(O, "weno5", 0.1, per, open_).advect_fct(*a, inflow=infl, flux_face_i=fi)
    np.testing.assert_array_equal(got, ref)
    np.testing.assert_array_equal(fx, rx)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_tracers_of_one_cta_equal_the_tracers_alone(precision):
    """A grid large enough for CTAs that take every tracer of a layer: each tracer as on its own."""
    nt, n, ny, nx = 3, 40, 133, 197
    C, V0, V1, Qx, Qy, ok = (torch.from_numpy(x).cuda() for x in _domain(3, nt, n, ny, nx, ()))
    adv = P.TracerAdvection(scheme="weno5", time="ssprk3", dt=0.1, precision=precision)
    got = adv.advect_fct(C, V0, V1, Qx, Qy, ok)
    for t in range(nt):
        assert torch.equal(got[t], adv.advect_fct(C[t:t + 1].contiguous(), V0, V1, Qx, Qy, ok)[0])
