"""Forms that the passes' other tests leave out: the one-pass limiter on axes periodic in y and on non-finite values and
tied signed zeros; masks that start off a word; several tracers of one CTA in the unlimited and the RK3 step."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import pyocean_b200 as P
from pyocean_b200 import workloads as W
from pyocean_b200.batch import Domain, DomainBatch
from pyocean_b200.step import ALETracerStep

pytestmark = pytest.mark.gpu


def _bits(t):
    return torch.where(t != t, torch.zeros_like(t), t).view(torch.int64), t != t


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(_bits(a), _bits(b)))


def _workloads(values):
    out = []
    for i, (nx, ny, n, per) in enumerate([(230, 200, 24, ("y",)), (200, 129, 30, ("x", "y")), (141, 100, 20, ()), (29, 65, 2, ("y",)),
                                          (5, 4, 2, ("x", "y")), (28, 16, 3, ("y",)), (6, 3, 1, ("x", "y"))]):
        w = W.basin(seed=i, nx=nx, ny=ny, n=n, nt=1) if nx > 50 else W.zstar_box(seed=i, nx=nx, ny=ny, n=n, nt=1)
        w.periodic, w.open = per, () if per else ("west", "north")
        rng = np.random.default_rng(i)
        if values == "ties":                                          # equal bounds of either sign among a few values
            w.C = rng.choice([0.0, -0.0, 1.0, -1.0], w.C.shape)
        elif values == "non-finite":
            w.C = w.C.copy()
            w.C[rng.random(w.C.shape) < 1e-3] = np.nan
            w.C[rng.random(w.C.shape) < 1e-3] = np.inf
            w.C[rng.random(w.C.shape) < 1e-3] = -np.inf
        out.append(w)
    return out


@pytest.mark.parametrize("values", ["plain", "ties", "non-finite"])
def test_one_pass_limiter(values):
    dev = torch.device("cuda", 0)
    ws = _workloads(values)
    doms = [Domain.from_workload(w, dev) for w in ws]
    assert sum(d.cells for d in doms) >= 1 << 21                      # the batch limits in one pass
    batch = DomainBatch(doms)
    batch.step(1)
    for i, (w, dom) in enumerate(zip(ws, doms)):
        st = ALETracerStep(*dom.shape, dom.dt, dom.flags, dom.remap_scheme, device=dev)
        c = torch.from_numpy(np.ascontiguousarray(w.C)).to(dev)
        assert _same(dom.C_adv, st.advect(c, dom.V0, dom.V1, dom.Qx, dom.Qy, dom.ok)), (i, dom.shape)


def _fields(nt, n, ny, nx):
    g = torch.Generator(device="cuda")
    g.manual_seed(nt * n + nx)
    r = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)       # noqa: E731
    V0 = 1.0 + r(n, ny, nx)
    Qx, Qy = 0.1 * (r(n, ny, nx + 1) - 0.5), 0.1 * (r(n, ny + 1, nx) - 0.5)
    return 10.0 + r(nt, n, ny, nx), V0, V0 * (1.0 + 0.01 * r(n, ny, nx)), Qx, Qy, r(n, ny, nx) > 0.1


@pytest.mark.parametrize("offset", [1, 2, 3, 5])
@pytest.mark.parametrize("nx", [7, 32, 64])
def test_masks_that_start_off_a_word(nx, offset):
    C, V0, V1, Qx, Qy, ok = _fields(2, 3, 19, nx)
    flat = torch.zeros(ok.numel() + 16, dtype=torch.bool, device="cuda")
    view = flat[offset:offset + ok.numel()].view(ok.shape)
    view.copy_(ok)
    adv = P.TracerAdvection(scheme="weno5", time="ssprk3", dt=1.0)
    Fz = torch.zeros((4, 19, nx), dtype=torch.float64, device="cuda")
    Fz[1:3] = 0.01
    h = V0.clone()
    for call in (lambda m: adv.advect_fct(C, V0, V1, Qx, Qy, m), lambda m: adv.advect(C, V0, V1, Qx, Qy, Fz, m),
                 lambda m: adv.rhs(C, Qx, Qy, Fz, m), lambda m: P.remap_columns(h, C, V1, P.PPM_H4, m[0])):
        assert _same(call(view), call(ok))


@pytest.mark.parametrize("kind", ["unlimited", "ssprk3", "pc"])
def test_tracers_of_one_cta(kind):
    """A grid large enough for CTAs that take every tracer of a layer: each tracer as on its own."""
    C, V0, V1, Qx, Qy, ok = _fields(3, 40, 133, 197)
    Fz = torch.zeros((41, 133, 197), dtype=torch.float64, device="cuda")
    Fz[1:40] = 0.01 * (V0[1:] - 1.5)
    adv = P.TracerAdvection(scheme="weno5", time="pc" if kind == "pc" else "ssprk3", dt=1.0)

    def step(c):
        if kind == "unlimited":
            return adv.advect_fct(c, V0, V1, Qx, Qy, ok, unlimited=True, flux_face_i=5)
        return adv.advect(c, V0, V1, Qx, Qy, Fz, ok, flux_face_i=5)

    got = step(C)
    for t in range(3):
        for a, b in zip(got, step(C[t:t + 1].contiguous())):
            assert torch.equal(a[t], b[0])
