"""What users of this framework have it compute, as cases that can be timed: the ALE tracer step and its parts, through
the public entry points, on device-resident fields.

Sizes come from the repository's own configurations (the 64 x 64 x 20 z* box, the 512 x 512 x 50 basin, uneven domains
of 96..384 cells, mixed precision on a deep basin) and from ragged regional grids between them; thicknesses, transports
and tracers have the distributions of ``pyocean_b200.workloads``, drawn on the device from the seed.

``exact`` evaluates each case in float64 with plain torch operations.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from pyocean_b200 import _lib, ale_tracer_step
from pyocean_b200.batch import Domain, DomainBatch
from pyocean_b200.diffusion import diffuse_ale
from pyocean_b200.periodic import Periodic
from pyocean_b200.producers import ALELayerTransport
from pyocean_b200.remap import remap_columns
from pyocean_b200.tracers import OpenEdges, TracerAdvection
from pyocean_b200.vertical import ALECoordinate

F64 = torch.float64
PCM, PLM, PPM = 0, 1, 2


def listed() -> list:
    return [
        # one step of a small process-study box, the smallest domain a user steps: launches and latency count
        dict(name="step_box_64", kind="step", box=True, nx=64, ny=64, n=20, nt=1, scheme=PPM),
        # the production step: T and S of the 512 x 512 x 50 basin, advected with the limiter and remapped
        dict(name="step_basin_512", kind="step", box=False, nx=512, ny=512, n=50, nt=2, scheme=PPM),
        # a regional grid with odd sizes, four open edges, exterior values and a section's tracer flux, three tracers
        dict(name="fct_regional_open", kind="fct", box=False, nx=333, ny=257, n=41, nt=3, precision="f64", open=True,
             js=False),
        # many tracers on a deep basin at reduced precision (T, S and top-hat passive tracers)
        dict(name="fct_mixed_deep", kind="fct", box=False, nx=512, ny=512, n=75, nt=4, precision="mixed", open=False,
             js=False),
        # the step without limiter, with a vertical transport through the layers (geopotential models)
        dict(name="advect_rk3_basin", kind="rk3", box=False, nx=384, ny=320, n=50, nt=2),
        # a stack of three tracers remapped between grids of different layer counts
        dict(name="remap_ppm_odd", kind="remap", nx=511, ny=389, n=60, n1=50, nt=3, scheme=PPM),
        # one field with the cheaper scheme on a small grid
        dict(name="remap_plm_small", kind="remap", nx=150, ny=121, n=30, n1=30, nt=1, scheme=PLM),
        # an ensemble of uneven boxes advanced together, two steps
        dict(name="batch_uneven_24", kind="batch", domains=24, lo=96, hi=384, nt=1, pick=0),
        # the vertical coordinate's own call: z* target grid and the remap of two tracers onto it
        dict(name="regrid_remap_zstar", kind="regrid", nx=400, ny=360, n=50, nt=2, scheme=PPM),
        # the layer transport that produces the step's fluxes and volumes (PPM thickness flux)
        dict(name="layer_transport_ppm", kind="layers", nx=512, ny=512, n=50),
        # lateral diffusion of two tracers along the layers
        dict(name="diffuse_basin", kind="diffuse", nx=512, ny=512, n=50, nt=2),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "fct", "fct", "rk3", "remap", "remap", "batch", "regrid", "layers", "diffuse"])
    while True:
        nx, ny, n, nt = _log(rng, 48, 640), _log(rng, 48, 640), _log(rng, 10, 75), rng.randint(1, 4)
        if nx * ny * n * nt <= 512 * 512 * 50 * 2:
            break
    if kind == "step":
        return dict(kind=kind, box=rng.random() < 0.4, nx=nx, ny=ny, n=n, nt=nt, scheme=rng.choice([PPM, PPM, PLM, PCM]))
    if kind == "fct":
        return dict(kind=kind, box=False, nx=nx, ny=ny, n=n, nt=nt, precision=rng.choice(["f64", "f64", "mixed"]),
                    open=rng.random() < 0.5, js=rng.random() < 0.25)
    if kind == "rk3":
        return dict(kind=kind, box=rng.random() < 0.4, nx=nx, ny=ny, n=n, nt=nt)
    if kind == "remap":
        return dict(kind=kind, nx=nx, ny=ny, n=n, n1=n if rng.random() < 0.6 else _log(rng, 10, 75), nt=nt,
                    scheme=rng.choice([PPM, PPM, PLM, PCM]))
    if kind == "batch":
        return dict(kind=kind, domains=rng.randint(3, 20), lo=48, hi=320, nt=rng.randint(1, 2), pick=rng.randint(0, 9999))
    if kind == "regrid":
        return dict(kind=kind, nx=nx, ny=ny, n=n, nt=nt, scheme=rng.choice([PPM, PLM]))
    if kind == "layers":
        return dict(kind=kind, nx=nx, ny=ny, n=n)
    return dict(kind=kind, nx=nx, ny=ny, n=n, nt=nt)


# ---------------------------------------------------------------------------------------------------------- inputs
class _Gen:
    """Seeded draws on the device."""

    def __init__(self, seed: int) -> None:
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) * 7919 + 17)

    def u(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, generator=self.g, dtype=F64, device="cuda")

    def n(self, scale, *shape):
        return scale * torch.randn(shape, generator=self.g, dtype=F64, device="cuda")


def _grid(ny: int, nx: int):
    y = torch.arange(ny, dtype=F64, device="cuda")[:, None]
    return y, torch.arange(nx, dtype=F64, device="cuda")[None, :]


def _blobs(gen: _Gen, ny: int, nx: int, count: int, rlo: float, rhi: float, by_radius: bool = False):
    """Sum of ``count`` Gaussian bumps of random sign and radius rlo..rhi cells (separable, so one product)."""
    y, x = _grid(ny, nx)
    cx, cy, r = gen.u(0, nx, count), gen.u(0, ny, count), gen.u(rlo, rhi, count)
    amp = gen.u(-1, 1, count) * (r if by_radius else 1.0)
    ey = torch.exp(-(y - cy[None, :]) ** 2 / (2 * r * r)[None, :])                     # (ny, count)
    ex = torch.exp(-(x - cx[:, None]) ** 2 / (2 * r * r)[:, None])                     # (count, nx)
    return (ey * amp[None, :]) @ ex


def _transports(psi, h, water, per_x: bool, open_edges: bool):
    """Divergence-free layer transports from a corner streamfunction; no transport touches land."""
    n, ny, nx = h.shape
    wp = torch.full((ny + 2, nx + 2), bool(open_edges), device="cuda")
    wp[1:-1, 1:-1] = water
    hp = torch.nn.functional.pad(h, (1, 1, 1, 1), mode="replicate")
    if per_x:
        wp[1:-1, 0], wp[1:-1, -1] = water[:, -1], water[:, 0]
        hp[:, 1:-1, 0], hp[:, 1:-1, -1] = h[:, :, -1], h[:, :, 0]
        psi = psi.clone()
        psi[:, -1] = psi[:, 0]
    m = wp[:-1, :-1] & wp[:-1, 1:] & wp[1:, :-1] & wp[1:, 1:]
    hc = 0.25 * (hp[:, :-1, :-1] + hp[:, :-1, 1:] + hp[:, 1:, :-1] + hp[:, 1:, 1:])
    if per_x:
        m[:, -1] = m[:, 0]
        hc[:, :, -1] = hc[:, :, 0]
    P = psi[None] * hc * m[None]
    return -(P[:, 1:, :] - P[:, :-1, :]), P[:, :, 1:] - P[:, :, :-1]


def _ocean(case: dict, seed: int) -> SimpleNamespace:
    """Geometry, transports and tracers of a basin (bathymetry, land, a hybrid grid, eddies) or of a z* box."""
    gen = _Gen(seed)
    nx, ny, n, nt = case["nx"], case["ny"], case["n"], case.get("nt", 1)
    box, opened = case.get("box", False), case.get("open", False)
    o = SimpleNamespace(per=("x",) if box else (), open=("west", "east", "south", "north") if opened else ())
    y, x = _grid(ny, nx)
    if box:
        dx = torch.full((ny, nx), 1000.0, dtype=F64, device="cuda")
        dy = dx.clone()
        water = torch.ones((ny, nx), dtype=torch.bool, device="cuda")
        H = torch.full((ny, nx), 5.0 * n, dtype=F64, device="cuda")
        h = torch.full((n, ny, nx), 5.0, dtype=F64, device="cuda")
        spread, umax = 0.2, 0.5
        m, kk = torch.arange(1, 9, dtype=F64, device="cuda"), torch.arange(-8, 9, dtype=F64, device="cuda")
        ph = gen.u(0, 2 * math.pi, 8, 17)
        amp = torch.hypot(m[:, None] / 2, kk[None, :]) ** -3
        ic, jc = torch.arange(nx + 1, dtype=F64, device="cuda") / nx, torch.arange(ny + 1, dtype=F64, device="cuda") / ny
        gx = (amp[..., None] * torch.cos(2 * math.pi * kk[None, :, None] * ic + ph[..., None])).sum(1)
        psi = torch.sin(math.pi * m[None, :] * jc[:, None]) @ gx
    else:
        dx = 2000.0 * (1 + 0.05 * torch.cos(2 * math.pi * (x / 70 + y / 90) + gen.u(0, 6, 1)))
        dy = 2000.0 * (1 + 0.05 * torch.cos(2 * math.pi * (x / 80 - y / 60) + gen.u(0, 6, 1)))
        bump = _blobs(gen, ny, nx, 40, 0.03 * nx, 0.15 * nx)
        bump = (bump - bump.min()) / (bump.max() - bump.min())
        H = 50.0 + 3950.0 * bump
        water = H > H.flatten().kthvalue(max(1, int(0.15 * nx * ny))).values
        if not opened:
            water[0, :] = water[-1, :] = False
            water[:, 0] = water[:, -1] = False
        H = torch.where(water, H, 0.0)
        ntop = n // 2                                  # z-like 10 m layers on top, stretched ones below
        top = torch.clamp(H / n, max=10.0)
        rest = torch.clamp(H - ntop * top, min=0.0)
        w = torch.linspace(2.0, 1.0, n - ntop, dtype=F64, device="cuda")
        h = torch.cat([(w / w.sum())[:, None, None] * rest, top.expand(ntop, ny, nx)])
        spread, umax = 0.3, 1.0
        psi = _blobs(gen, ny + 1, nx + 1, 60, 8.0, 40.0, by_radius=True)
    area = dx * dy
    Qx, Qy = _transports(psi, h, water, box, opened)
    hx = torch.cat([h[..., :1], 0.5 * (h[..., 1:] + h[..., :-1]), h[..., -1:]], -1)
    hy = torch.cat([h[:, :1], 0.5 * (h[:, 1:] + h[:, :-1]), h[:, -1:]], 1)
    fast = max(float((Qx.abs() / (950.0 * hx)).nan_to_num(0, 0, 0).max()),
               float((Qy.abs() / (950.0 * hy)).nan_to_num(0, 0, 0).max())) * (1.0 if box else 0.5)
    Qx, Qy = Qx * (umax / fast), Qy * (umax / fast)
    o.dt = 0.4 * (1000.0 if box else 1900.0) / umax
    V0 = area * h
    V1 = V0 - o.dt * (Qx[..., 1:] - Qx[..., :-1] + Qy[:, 1:] - Qy[:, :-1])
    o.V0, o.V1, o.Qx, o.Qy, o.ok, o.wet = V0, V1, Qx, Qy, water & (V1 > 0), water
    o.H, o.h_tgt, o.area, o.dx, o.dy = H, h, area, dx, dy
    hs = h * (1 + gen.u(-spread, spread, n, ny, nx))
    col = hs.sum(0)
    o.h_src = hs * torch.where(col > 0, h.sum(0) / torch.where(col > 0, col, 1.0), 0.0)
    o.gen = gen
    if "nt" in case:
        C = torch.empty((nt, n, ny, nx), dtype=F64, device="cuda")
        if box:
            C[:] = torch.where(torch.arange(nx, device="cuda") < nx // 2, 10.0, 20.0) + gen.n(0.01, nt, n, ny, nx)
        else:
            frac = torch.clamp((H - (torch.cumsum(h, 0) - 0.5 * h)) / 4000.0, 0, 1)
            for t in range(nt):
                eddy = _blobs(gen, ny, nx, 30, 5.0, 30.0).clamp(-1, 1)
                if t == 0:
                    C[t] = 25.0 - 21.0 * frac + eddy
                elif t == 1:
                    C[t] = 34.0 + frac + 0.1 * eddy
                else:                                  # a patch of 1 in a field of 0, over part of the column
                    k0 = int(float(gen.u(0, 0.7 * n, 1)))
                    C[t] = 0.0
                    C[t, k0:k0 + max(1, n // 4)] = (eddy > 0.2).to(F64)
        o.C = C
    return o


def _layer_inputs(case: dict, seed: int) -> SimpleNamespace:
    """The velocities, face thicknesses and weights the layer transport is called with."""
    o = _ocean(case, seed)
    gen, n = o.gen, case["n"]
    act, h = o.wet, torch.where(o.wet, o.h_src, 0.0)
    o.h, o.dt = h, 300.0
    hx, hy = 0.5 * (h[..., 1:] + h[..., :-1]), 0.5 * (h[:, 1:] + h[:, :-1])
    o.wet_u, o.wet_v = torch.zeros_like(o.Qx[0], dtype=torch.bool), torch.zeros_like(o.Qy[0], dtype=torch.bool)
    o.wet_u[:, 1:-1], o.wet_v[1:-1] = act[:, 1:] & act[:, :-1], act[1:] & act[:-1]
    Hs = h.sum(0)
    o.H = Hs
    o.Du, o.Dv = torch.zeros_like(o.Qx[0]), torch.zeros_like(o.Qy[0])
    o.Du[:, 1:-1], o.Dv[1:-1] = torch.minimum(Hs[:, 1:], Hs[:, :-1]), torch.minimum(Hs[1:], Hs[:-1])
    u, v = torch.zeros_like(o.Qx), torch.zeros_like(o.Qy)
    u[..., 1:-1] = (o.Qx[..., 1:-1] / (2000.0 * hx)).nan_to_num(0, 0, 0).clamp(-1, 1)
    v[:, 1:-1] = (o.Qy[:, 1:-1] / (2000.0 * hy)).nan_to_num(0, 0, 0).clamp(-1, 1)
    o.u0, o.v0 = (u + gen.n(0.02, *u.shape)) * o.wet_u, (v + gen.n(0.02, *v.shape)) * o.wet_v
    o.u1, o.v1 = (u + gen.n(0.02, *u.shape)) * o.wet_u, (v + gen.n(0.02, *v.shape)) * o.wet_v
    o.qe, o.qw = _face_thickness(h, Hs, act)
    qn, qs = _face_thickness(h.transpose(1, 2), Hs.T, act.T)
    o.qn, o.qs = qn.contiguous(), qs.contiguous()                     # v-faces on swapped axes, as the call takes them
    frac = lambda a: torch.where(a.sum(0) > 0, a / a.sum(0).clamp(min=1e-300), 1.0 / n)               # noqa: E731
    o.wu = frac(0.5 * (o.qe + o.qw))
    o.wv = frac(0.5 * (o.qn + o.qs)).transpose(1, 2).contiguous()
    o.Lu, o.Lv = torch.full_like(o.Du, 2000.0), torch.full_like(o.Dv, 2000.0)
    return o


def _face_thickness(h, H, act):
    """Layer thickness available on each u-face from its west and east cell, above the shallower bed."""
    n, ny, nx = h.shape
    iw, ie = torch.arange(-1, nx, device="cuda").clamp(min=0), torch.arange(nx + 1, device="cuda").clamp(max=nx - 1)
    bed = torch.maximum(-H[:, iw], -H[:, ie])
    open_ = act[:, iw] & act[:, ie]
    top = -H + torch.cumsum(h, 0)
    q = [torch.where(open_, torch.minimum(h[..., s], (top[..., s] - bed).clamp(min=0.0)), 0.0) for s in (iw, ie)]
    return q[0].contiguous(), q[1].contiguous()


def _box_sizes(case: dict) -> list:
    """(nx, ny, n) of the batch's domains: nx, ny log-uniform in lo..hi, n of 30, 50, 75 (the same for every seed)."""
    g = torch.Generator().manual_seed(1000 + case["pick"])
    r = torch.rand((case["domains"], 3), generator=g, dtype=F64)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [(int(round(math.exp(lo + float(a) * (hi - lo)))), int(round(math.exp(lo + float(b) * (hi - lo)))),
             (30, 50, 75)[min(2, int(float(c) * 3))]) for a, b, c in r]


def _boxes(case: dict, seed: int) -> list:
    return [_ocean(dict(box=True, nx=nx, ny=ny, n=n, nt=case["nt"]), seed * 100 + d)
            for d, (nx, ny, n) in enumerate(_box_sizes(case))]


def _remap_inputs(case: dict, seed: int) -> SimpleNamespace:
    """Lagrangian source layers and a target of n1 layers of the same columns; fields with fronts in the vertical."""
    o = _ocean(dict(case, box=False), seed)
    gen, n1, n, nt = o.gen, case["n1"], case["n"], case["nt"]
    C = o.C + gen.n(0.02, *o.C.shape)                                 # as rough as advected fields
    w = 1.0 + 0.5 * torch.cos(torch.linspace(0, 3, n1, dtype=F64, device="cuda"))
    o.C = C
    if n1 != n:
        o.h_tgt = (w / w.sum())[:, None, None] * o.h_src.sum(0)
    return o


def _fz(o, case: dict):
    n, ny, nx = case["n"], case["ny"], case["nx"]
    Fz = torch.zeros((n + 1, ny, nx), dtype=F64, device="cuda")
    Fz[1:-1] = o.gen.n(100.0, n - 1, ny, nx) * o.wet
    return Fz


def _diffusion_inputs(case: dict, seed: int) -> SimpleNamespace:
    o = _ocean(dict(case, box=False), seed)
    gen, ny, nx = o.gen, case["ny"], case["nx"]
    o.cx, o.cy = gen.u(0.9, 1.1, ny, nx + 1), gen.u(0.9, 1.1, ny + 1, nx)
    o.okx, o.oky = gen.u(0, 1, ny, nx + 1) > 0.02, gen.u(0, 1, ny + 1, nx) > 0.02
    o.Tw = o.C - 10.0
    return o


# ------------------------------------------------------------------------------------------------- prepare and run
def _advection(case: dict, o) -> TracerAdvection:
    adv = TracerAdvection(scheme="weno5js" if case.get("js") else "weno5", time="ssprk3", dt=o.dt, ob=OpenEdges(o.open),
                          precision=case.get("precision", "f64"))
    adv.per = Periodic(o.per)
    return adv


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("step", "fct", "rk3"):
        o = _ocean(case, seed)
        s = SimpleNamespace(case=case, o=o, adv=_advection(case, o))
        if kind == "fct" and case["open"]:
            s.inflow = o.C + o.gen.n(0.2, *o.C.shape)
        if kind == "rk3":
            s.Fz = _fz(o, case)
    elif kind == "remap":
        s = SimpleNamespace(case=case, o=_remap_inputs(case, seed))
    elif kind == "batch":
        boxes = _boxes(case, seed)
        flags = _lib.PERIODIC_X
        doms = [Domain.from_tensors(b.C, b.V0, b.V1, b.Qx, b.Qy, b.ok.to(torch.uint8), b.h_src, b.h_tgt,
                                    b.wet.to(torch.uint8), flags, b.dt, PPM) for b in boxes]
        s = SimpleNamespace(case=case, start=[b.C for b in boxes], batch=DomainBatch(doms))
    elif kind == "regrid":
        o = _ocean(dict(case, box=False), seed)
        o.eta = 0.3 * _blobs(o.gen, case["ny"], case["nx"], 20, 10.0, 40.0).clamp(-1, 1)
        dz = torch.full((case["n"],), 4000.0 / case["n"], dtype=F64).numpy()
        s = SimpleNamespace(case=case, o=o, coord=ALECoordinate(o.H, o.wet, "zstar", dict(dz_top=dz), case["scheme"]))
    elif kind == "layers":
        o = _layer_inputs(case, seed)
        fs = SimpleNamespace(theta=0.6, active=o.wet, Lu=o.Lu, Lv=o.Lv)
        s = SimpleNamespace(case=case, o=o, st=SimpleNamespace(h=o.h, u=o.u0, v=o.v0, eta=None),
                            fl=SimpleNamespace(wet_u=o.wet_u, wet_v=o.wet_v, Du=o.Du, Dv=o.Dv, fw=None),
                            lt=ALELayerTransport(fs=fs, H=o.H, area=o.area, dt=o.dt, thickness_flux="ppm",
                                                 vi_geom=dict(dx_t=o.dx, dy_t=o.dy)))
    else:
        s = SimpleNamespace(case=case, o=_diffusion_inputs(case, seed))
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "step":
        o = s.o
        return ale_tracer_step(s.adv, o.C, o.V0, o.V1, o.Qx, o.Qy, o.ok, o.h_src, o.h_tgt, s.case["scheme"], o.wet)
    if kind == "fct":
        o = s.o
        if s.case["open"]:
            return s.adv.advect_fct(o.C, o.V0, o.V1, o.Qx, o.Qy, o.ok, inflow=s.inflow, flux_face_i=s.case["nx"] // 2)
        return s.adv.advect_fct(o.C, o.V0, o.V1, o.Qx, o.Qy, o.ok)
    if kind == "rk3":
        o = s.o
        return s.adv.advect(o.C, o.V0, o.V1, o.Qx, o.Qy, s.Fz, o.ok)
    if kind == "remap":
        o = s.o
        return remap_columns(o.h_src, o.C, o.h_tgt, s.case["scheme"], o.wet)
    if kind == "batch":
        b = s.batch
        for i, c in enumerate(s.start):                # this ensemble's fields go into the resident domains
            b.state(i).copy_(c)
        b.step(2)
        return [b.state(i) for i in range(len(s.start))]
    if kind == "regrid":
        h_new, outs = s.coord.regrid_remap(s.o.eta, s.o.h_src, s.o.C)
        return h_new, outs
    if kind == "layers":
        o = s.o
        f = s.lt(s.st, None, o.u1, o.v1, s.fl, 0.5, (), o.wu, o.wv, o.qe, o.qw, o.qn, o.qs)
        return dict(Qx=f.Qx, Qy=f.Qy, V0=f.V0, V1=f.V1, ok=f.ok, h_dagger=f.h_dagger)
    o = s.o
    return diffuse_ale(o.C, o.Tw, o.h_tgt, o.wet, o.cx, o.cy, o.okx, o.oky, o.V0, 100.0, 600.0)


# --------------------------------------------------------------------------------------------------- bytes and work
# FP64 operations of the method per item: a WENO5 face value, a limited cell, a remapped cell, a PPM layer flux
_FACE, _LIMIT, _REMAP, _PPM_FLUX = 75, 90, 110, 25


def _step_work(n: int, ny: int, nx: int, nt: int, what: str) -> dict:
    cells, faces = n * ny * nx, n * (2 * ny * nx + ny + nx)
    adv = dict(bytes=cells * (16 * nt + 17) + 8 * faces, flops=nt * (3 * faces * _FACE + cells * _LIMIT))
    rem = dict(bytes=cells * (16 + 16 * nt) + ny * nx, flops=nt * cells * _REMAP)
    if what == "fct":
        return adv
    return dict(bytes=adv["bytes"] + rem["bytes"], flops=adv["flops"] + rem["flops"])


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        w = [_step_work(n, ny, nx, case["nt"], "step") for nx, ny, n in _box_sizes(case)]
        return {k: 2 * sum(x[k] for x in w) for k in ("bytes", "flops")}
    nx, ny, n, nt = case["nx"], case["ny"], case["n"], case.get("nt", 1)
    cells, plane = n * ny * nx, ny * nx
    if kind == "step":
        return _step_work(n, ny, nx, nt, "step")
    if kind == "fct":
        w = _step_work(n, ny, nx, nt, "fct")
        extra = 8 * nt * n * ny if case["open"] else 0               # the section's flux
        edges = 8 * nt * n * 2 * (ny + nx) if case["open"] else 0    # exterior values, read on the edges only
        return dict(bytes=w["bytes"] + extra + edges, flops=w["flops"])
    if kind == "rk3":
        faces = n * (3 * plane + ny + nx)
        return dict(bytes=cells * (16 * nt + 17) + 8 * faces, flops=nt * (3 * faces * _FACE + cells * 30))
    if kind == "remap":
        n1 = case["n1"]
        return dict(bytes=8 * plane * (n + n1) * (1 + nt) + plane, flops=nt * plane * max(n, n1) * _REMAP)
    if kind == "regrid":
        return dict(bytes=cells * (16 + 16 * nt) + 18 * plane, flops=nt * cells * _REMAP + 6 * cells)
    if kind == "layers":                               # h, u and v twice, weights, face thicknesses; fluxes, volumes
        return dict(bytes=8 * cells * 17 + cells, flops=2 * 22 * cells * _PPM_FLUX)
    return dict(bytes=cells * (24 * nt + 16) + 19 * plane, flops=20 * nt * cells)


# ------------------------------------------------------------------------------------------------------------ exact
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "step":
        o = _ocean(case, seed)
        return _remap(o.h_src, _fct(case, o), o.h_tgt, case["scheme"], o.wet)
    if kind == "fct":
        o = _ocean(case, seed)
        if not case["open"]:
            return _fct(case, o)
        return _fct(case, o, inflow=o.C + o.gen.n(0.2, *o.C.shape), section=case["nx"] // 2)
    if kind == "rk3":
        o = _ocean(case, seed)
        return _rk3(case, o, _fz(o, case))
    if kind == "remap":
        o = _remap_inputs(case, seed)
        return _remap(o.h_src, o.C, o.h_tgt, case["scheme"], o.wet)
    if kind == "batch":
        out = []
        for b in _boxes(case, seed):
            for _ in range(2):
                b.C = _remap(b.h_src, _fct({}, b), b.h_tgt, PPM, b.wet)
            out.append(b.C)
        return out
    if kind == "regrid":
        o = _ocean(dict(case, box=False), seed)
        eta = 0.3 * _blobs(o.gen, case["ny"], case["nx"], 20, 10.0, 40.0).clamp(-1, 1)
        h_new, wet = _zstar(o, eta, case["n"])
        return h_new, _remap(o.h_src, o.C, h_new, case["scheme"], wet)
    if kind == "layers":
        return _layer_transport(_layer_inputs(case, seed))
    o = _diffusion_inputs(case, seed)
    return _diffuse(o, 100.0, 600.0)


def _weno(v1, v2, v3, v4, v5, all5, mid3, z: bool):
    """WENO5 (Z or JS weights) of an upwind-ordered stencil; WENO3 or the upwind cell where cells are missing."""
    q0 = (2 * v1 - 7 * v2 + 11 * v3) / 6
    q1 = (-v2 + 5 * v3 + 2 * v4) / 6
    q2 = (2 * v3 + 5 * v4 - v5) / 6
    b0 = 13 / 12 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2
    b1 = 13 / 12 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2
    b2 = 13 / 12 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2
    if z:
        tau = (b2 - b0).abs()
        a = [d * (1 + tau / (1e-40 + b)) for d, b in ((0.1, b0), (0.6, b1), (0.3, b2))]
    else:
        a = [d / (1e-6 + b) ** 2 for d, b in ((0.1, b0), (0.6, b1), (0.3, b2))]
    five = (a[0] * q0 + a[1] * q1 + a[2] * q2) / (a[0] + a[1] + a[2])
    e0, e1 = 1 / 3 / (1e-6 + (v3 - v2) ** 2) ** 2, 2 / 3 / (1e-6 + (v4 - v3) ** 2) ** 2
    three = (e0 * (-v2 + 3 * v3) / 2 + e1 * (v3 + v4) / 2) / (e0 + e1)
    return torch.where(all5, five, torch.where(mid3, three, v3))


def _face_flux(c, Q, ok, ext, per: bool, lo: bool, hi: bool, z: bool):
    """Q times the WENO face value on every face of the last axis of c (n, ny, nx); Q has one more entry."""
    nx = c.shape[-1]
    if per:
        Q = torch.cat([Q[..., :-1], Q[..., :1]], -1)
        idx = torch.arange(-3, nx + 3, device="cuda") % nx
        cp, kp = c[..., idx], ok[..., idx]
    else:
        cp, kp = torch.nn.functional.pad(c, (3, 3)), torch.nn.functional.pad(ok, (3, 3))
    w = [cp[..., m:m + nx + 1] for m in range(6)]
    k = [kp[..., m:m + nx + 1] for m in range(6)]
    pos = Q >= 0
    v = [torch.where(pos, w[m], w[5 - m]) for m in range(5)]
    kk = [torch.where(pos, k[m], k[5 - m]) for m in range(5)]
    mid = kk[1] & kk[2] & kk[3]
    F = torch.where(Q != 0, Q * _weno(*v, mid & kk[0] & kk[4], mid, z), 0.0)
    if not per:
        F[..., 0] = Q[..., 0] * torch.where(Q[..., 0] > 0, ext[..., 0], c[..., 0]) if lo else 0.0
        F[..., -1] = Q[..., -1] * torch.where(Q[..., -1] < 0, ext[..., -1], c[..., -1]) if hi else 0.0
    return F


def _donor_flux(c, Q, ext, per: bool, lo: bool, hi: bool):
    if per:
        Q = torch.cat([Q[..., :-1], Q[..., :1]], -1)
        w, e = torch.cat([c[..., -1:], c], -1), torch.cat([c, c[..., :1]], -1)
        return Q * torch.where(Q >= 0, w, e)
    F = torch.zeros_like(Q)
    q = Q[..., 1:-1]
    F[..., 1:-1] = q * torch.where(q >= 0, c[..., :-1], c[..., 1:])
    if lo:
        F[..., 0] = Q[..., 0] * torch.where(Q[..., 0] > 0, ext[..., 0], c[..., 0])
    if hi:
        F[..., -1] = Q[..., -1] * torch.where(Q[..., -1] < 0, ext[..., -1], c[..., -1])
    return F


def _tr(a):
    return a.transpose(-1, -2)


def _fct(case: dict, o, inflow=None, section=None):
    """SSP-RK3 WENO5 with Zalesak's limiter, one tracer at a time."""
    z, px, py = not case.get("js", False), "x" in o.per, "y" in o.per
    W, E, S, N = ("west" in o.open, "east" in o.open, "south" in o.open, "north" in o.open)
    outs, secs = [], []
    for t in range(o.C.shape[0]):
        C = o.C[t]
        ext = lambda c: c if inflow is None else inflow[t]                                            # noqa: E731
        div = lambda f: f[0][..., 1:] - f[0][..., :-1] + f[1][..., 1:, :] - f[1][..., :-1, :]          # noqa: E731
        safe = lambda q, V: torch.where(V > 0, q / torch.where(V > 0, V, 1.0), C)                      # noqa: E731

        def faces(c):
            fx = _face_flux(c, o.Qx, o.ok, ext(c), px, W, E, z)
            return fx, _tr(_face_flux(_tr(c), _tr(o.Qy), _tr(o.ok), _tr(ext(c)), py, S, N, z))

        q0, dV = o.V0 * C, o.V1 - o.V0
        f0 = faces(C)
        q1 = q0 - o.dt * div(f0)
        f1 = faces(safe(q1, o.V0 + dV))
        q2 = 0.75 * q0 + 0.25 * (q1 - o.dt * div(f1))
        f2 = faces(safe(q2, o.V0 + 0.5 * dV))
        lo = (_donor_flux(C, o.Qx, ext(C), px, W, E), _tr(_donor_flux(_tr(C), _tr(o.Qy), _tr(ext(C)), py, S, N)))
        A = [(a + b) / 6 + 2 * c / 3 - d for a, b, c, d in zip(f0, f1, f2, lo)]
        del f0, f1, f2, q1, q2
        cL = safe(q0 - o.dt * div(lo), o.V1)
        up, dn = torch.maximum(C, cL), torch.minimum(C, cL)
        up, dn = torch.where(o.ok, up, -math.inf), torch.where(o.ok, dn, math.inf)
        mx, mn = up.clone(), dn.clone()
        for ax, per in ((2, px), (1, py), (0, False)):
            for sh in (1, -1):
                for src, acc, fill in ((up, mx, -math.inf), (dn, mn, math.inf)):
                    r = torch.roll(src, sh, ax)
                    if not per:
                        r.select(ax, 0 if sh == 1 else r.shape[ax] - 1).fill_(fill)
                    if acc is mx:
                        mx = torch.maximum(mx, r)
                    else:
                        mn = torch.minimum(mn, r)
        pw, pe, ps, pn = A[0][..., :-1], A[0][..., 1:], A[1][..., :-1, :], A[1][..., 1:, :]
        p = lambda a: a.clamp(min=0.0)                                                                # noqa: E731
        Pin, Pout = o.dt * (p(pw) + p(-pe) + p(ps) + p(-pn)), o.dt * (p(pe) + p(-pw) + p(pn) + p(-ps))
        ratio = lambda q, P: torch.where(o.ok & (P > 0), (q.clamp(min=0) / torch.where(P > 0, P, 1.0)).clamp(max=1), 0.0)  # noqa: E731,E501
        Rp, Rm = ratio(o.V1 * (mx - cL), Pin), ratio(o.V1 * (cL - mn), Pout)

        def limited(A, Rp, Rm, per):
            c = torch.zeros_like(A)
            if per:
                l, r = torch.arange(-1, A.shape[-1] - 1, device="cuda") % (A.shape[-1] - 1), \
                    torch.arange(A.shape[-1], device="cuda") % (A.shape[-1] - 1)
                return torch.where(A >= 0, torch.minimum(Rp[..., r], Rm[..., l]), torch.minimum(Rp[..., l], Rm[..., r]))
            c[..., 1:-1] = torch.where(A[..., 1:-1] >= 0, torch.minimum(Rp[..., 1:], Rm[..., :-1]),
                                       torch.minimum(Rp[..., :-1], Rm[..., 1:]))
            return c

        F = (lo[0] + limited(A[0], Rp, Rm, px) * A[0], lo[1] + _tr(limited(_tr(A[1]), _tr(Rp), _tr(Rm), py)) * A[1])
        outs.append(safe(q0 - o.dt * div(F), o.V1))
        if section is not None:
            secs.append(F[0][..., section])
    return torch.stack(outs) if section is None else (torch.stack(outs), torch.stack(secs))


def _rk3(case: dict, o, Fz):
    """SSP-RK3 with WENO5-Z faces in x, y and z, no limiter."""
    px = "x" in o.per
    outs = []
    for t in range(o.C.shape[0]):
        C = o.C[t]
        safe = lambda q, V: torch.where(V > 0, q / torch.where(V > 0, V, 1.0), C)                      # noqa: E731

        def rhs(c):
            fx = _face_flux(c, o.Qx, o.ok, c, px, False, False, True)
            fy = _tr(_face_flux(_tr(c), _tr(o.Qy), _tr(o.ok), _tr(c), False, False, False, True))
            up = lambda a: a.movedim(0, -1)                                                            # noqa: E731
            fz = _face_flux(up(c), up(Fz), up(o.ok), up(c), False, False, False, True).movedim(-1, 0)
            return -(fx[..., 1:] - fx[..., :-1] + fy[..., 1:, :] - fy[..., :-1, :] + fz[1:] - fz[:-1])

        q0, dV = o.V0 * C, o.V1 - o.V0
        q1 = q0 + o.dt * rhs(C)
        q2 = 0.75 * q0 + 0.25 * (q1 + o.dt * rhs(safe(q1, o.V0 + dV)))
        q = q0 / 3 + 2 / 3 * (q2 + o.dt * rhs(safe(q2, o.V0 + 0.5 * dV)))
        outs.append(safe(q, o.V1))
    return torch.stack(outs)


def _sgn(x):
    return torch.where(x >= 0, 1.0, -1.0).to(F64)


def _plm(h, u):
    """Piecewise linear reconstruction (limited slopes, then monotone edges): c0, c1 of every cell of (n, P)."""
    n, eps = h.shape[0], 2.220446049250313e-16
    slp, mslp = torch.zeros_like(u), torch.zeros_like(u)
    l, c, r = u[:-2], u[1:-1], u[2:]
    sc = 2 * (r - l) * (h[1:-1] / (h[:-2] + 2 * h[1:-1] + h[2:] + 1e-30))
    lo, hi = torch.minimum(torch.minimum(l, c), r), torch.maximum(torch.maximum(l, c), r)
    s = torch.where((c - l) * (r - c) > 0, _sgn(sc) * torch.minimum(sc.abs(), 2 * torch.minimum(c - lo, hi - c)), 0.0)
    s = torch.where((c - 0.5 * s.abs() < lo) | (c + 0.5 * s.abs() > hi), s * (1 - eps), s)
    slp[1:-1] = torch.where(s.abs() < 1e-140, 0.0, s)
    er, el = l + 0.5 * slp[:-2], r - 0.5 * slp[2:]
    m = slp[1:-1].abs()
    a, b = c - 0.5 * slp[1:-1], c + 0.5 * slp[1:-1]
    m = torch.where((a - er) * (c - a) < 0, torch.minimum(m, (0.5 * (a + er) - c).abs() * 2 * (1 - eps)), m)
    m = torch.where((b - c) * (el - b) < 0, torch.minimum(m, (0.5 * (b + el) - c).abs() * 2 * (1 - eps)), m)
    mslp[1:-1] = _sgn(slp[1:-1]) * m
    c0, c1 = u.clone(), torch.zeros_like(u)
    c0[1:-1] = c - 0.5 * mslp[1:-1]
    d = (c + 0.5 * mslp[1:-1]) - c0[1:-1]
    e = d + c0[1:-1]
    en = u[2:] - 0.5 * _sgn(slp[2:]) * mslp[2:].abs()
    c1[1:-1] = torch.where((e - c) * (en - e) < 0, d * (1 - eps), d)
    return c0, c1, torch.zeros_like(u)


def _end_cubic(h, u):
    """Value at the end and at the first inner edge of the cubic with the means of the four end cells."""
    h1, h2, h3, h4 = (torch.clamp(a, min=1e-10) for a in h)
    h3 = torch.where(h2 + h3 < 1e-6 * h1, 1e-6 * h1 - h2, h3)
    h4 = torch.where(h3 + h4 < 1e-6 * h1, 1e-6 * h1 - h3, h4)
    # Newton's form of the primitive through the edges 0, h1, h1+h2, ...: its derivative at 0 and at h1
    x = [torch.zeros_like(h1), h1, h1 + h2, h1 + h2 + h3, h1 + h2 + h3 + h4]
    d = [u[0], u[1], u[2], u[3]]                                      # first divided differences
    d2 = [(d[i + 1] - d[i]) / (x[i + 2] - x[i]) for i in range(3)]
    d3 = [(d2[i + 1] - d2[i]) / (x[i + 3] - x[i]) for i in range(2)]
    d4 = (d3[1] - d3[0]) / (x[4] - x[0])

    def deriv(p):
        a, b, c, e = p - x[0], p - x[1], p - x[2], p - x[3]
        return d[0] + d2[0] * (a + b) + d3[0] * (a * b + a * c + b * c) + d4 * (a * b * c + a * b * e + a * c * e + b * c * e)

    return deriv(x[0]), deriv(x[1])


def _ppm(h, u):
    """PPM with explicit fourth-order edges, edge bounding and the Colella-Woodward limiter: c0, c1, c2."""
    n, eps = h.shape[0], 2.220446049250313e-16
    edge = torch.zeros((n + 1,) + h.shape[1:], dtype=F64, device="cuda")
    H = [h[:-3], h[1:-2], h[2:-1], h[3:]]
    U = [u[:-3], u[1:-2], u[2:-1], u[3:]]
    bad = (H[0] + H[1] == 0) | (H[1] + H[2] == 0) | (H[2] + H[3] == 0)
    floor = 1e-5 * torch.clamp(H[0] + H[1] + H[2] + H[3], min=1e-10)
    h0, h1, h2, h3 = (torch.where(bad, torch.maximum(floor, a), a) for a in H)
    i12, et2, et3 = 1 / (h1 + h2), 1 / ((h0 + h1 + h2) * (h0 + h1)), 1 / ((h1 + h2 + h3) * (h2 + h3))
    i012, i123 = (h0 + h1) * et2, (h2 + h3) * et3
    e = ((1 + (h1 * i012 + (h0 + h1) * i123)) * i12 * (h2 * (h2 + h3)) * U[1]
         + (1 + (h2 * i123 + (h2 + h3) * i012)) * i12 * (h1 * (h0 + h1)) * U[2]
         + (h1 * (h2 * (h2 + h3)) * et2 * (U[1] - U[0]) + h2 * (h1 * (h0 + h1)) * et3 * (U[2] - U[3])))
    edge[2:n - 1] = e / ((h0 + h1) + (h2 + h3))
    edge[0], edge[1] = _end_cubic(h[:4], u[:4])
    edge[n], edge[n - 1] = _end_cubic(h.flip(0)[:4], u.flip(0)[:4])
    el, er = edge[:-1].clone(), edge[1:].clone()
    um, up = torch.cat([u[:1], u[:-1]]), torch.cat([u[1:], u[-1:]])
    hm, hp = torch.cat([h[:1], h[:-1]]), torch.cat([h[1:], h[-1:]])
    den = hm + hp + 2 * h
    sl, sr, sc = u - um, up - u, torch.where(den > 0, (up - um) * (h / torch.where(den > 0, den, 1.0)), 0.0)
    s = torch.where((sl * sr > 0) & (den > 0),
                    _sgn(sc) * torch.minimum(torch.minimum(sl.abs(), sc.abs()), sr.abs()), 0.0)
    sg = _sgn(s)
    el = torch.where((um - el) * (el - u) < 0, u - sg * torch.minimum(s.abs(), (el - u).abs()), el)
    er = torch.where((up - er) * (er - u) < 0, u + sg * torch.minimum(s.abs(), (er - u).abs()), er)
    between = lambda e, a, b: torch.maximum(torch.minimum(e, torch.maximum(a, b)), torch.minimum(a, b))    # noqa: E731
    el, er = between(el, um, u), between(er, up, u)
    mid = between(0.5 * (er[:-1] + el[1:]), u[:-1], u[1:])
    jump = (el[1:] - er[:-1]) * (u[1:] - u[:-1]) < 0
    er[:-1], el[1:] = torch.where(jump, mid, er[:-1]), torch.where(jump, mid, el[1:])
    flat = (up - u) * (u - um) <= 0
    x1, x2 = 3 * (er - el) * ((u - el) + (u - er)), (er - el) ** 2
    el2, er2 = between(u + 2 * (u - er), um, u), between(u + 2 * (u - el), up, u)
    left, right = x1 > x2, (x1 <= x2) & (x1 < -x2)
    el, er = torch.where(flat, u, torch.where(left, el2, el)), torch.where(flat, u, torch.where(right, er2, er))
    same = (er - el).abs() < torch.clamp(eps * u.abs(), min=1e-60)
    el, er = torch.where(same, u, el), torch.where(same, u, er)
    c0, c1, c2 = el, 4 * (u - el) + 2 * (u - er), 3 * ((er - u) + (el - u))
    for c, v in ((c0, u), (c1, 0 * u), (c2, 0 * u)):
        c[0], c[-1] = v[0], v[-1]
    return c0, c1, c2


def _remap(h_src, C, h_tgt, scheme: int, wet):
    """Conservative remap of every wet column (every layer of a wet column here has water); others are copied, or NaN
    when the layer counts differ."""
    nt, n0, ny, nx = C.shape
    n1 = h_tgt.shape[0]
    w = wet.flatten()
    hs, ht = h_src.reshape(n0, -1)[:, w], h_tgt.reshape(n1, -1)[:, w]
    t1 = torch.cumsum(ht, 0)
    t0 = t1 - ht
    t0[1:] = t1[:-1]
    s1 = torch.cumsum(hs, 0)
    t1 = t1.clone()
    t1[-1] = torch.maximum(t1[-1], s1[-1])
    out = C.reshape(nt, n0, -1).clone() if n0 == n1 else torch.full((nt, n1, ny * nx), math.nan, dtype=F64, device="cuda")
    for m in range(nt):
        u = C[m].reshape(n0, -1)[:, w]
        if scheme == PPM and n0 >= 4:
            c0, c1, c2 = _ppm(hs, u)
        elif scheme >= PLM and n0 >= 3:
            c0, c1, c2 = _plm(hs, u)
        else:
            c0, c1, c2 = u, 0 * u, 0 * u
        content = torch.zeros_like(ht)
        for i in range(n0):
            a, b, hi = (s1[i - 1] if i else torch.zeros_like(s1[0])), s1[i], hs[i]
            lo, up = torch.maximum(t0, a), torch.minimum(t1, b)
            L = (up - lo).clamp(min=0)
            xa, xb = (lo - a) / hi, (up - a) / hi
            piece = L * (c0[i] + 0.5 * c1[i] * (xa + xb) + c2[i] * (xa * xa + xa * xb + xb * xb) / 3)
            piece = torch.where(L > 0, piece, 0.0)
            thick = L.argmax(0, keepdim=True)                         # takes what the others leave of the cell's content
            rest = u[i] * hi - (piece.sum(0) - piece.gather(0, thick)[0])
            content += piece.scatter(0, thick, rest[None])
        out[m][:, w] = content / ht
    return out.reshape(nt, n1, ny, nx)


def _zstar(o, eta, n: int):
    D = o.H + eta
    wet = o.wet & (D > 0) & (o.h_src.sum(0) > 0)
    hm, s = torch.clamp(D / n, max=1e-3), D / torch.where(o.H > 0, o.H, 1.0)
    e = [eta]
    for _ in range(n):
        e.append(e[-1] - s * (4000.0 / n))
    e[n] = -o.H
    for k in range(n - 1, -1, -1):
        e[k] = torch.maximum(e[k], e[k + 1] + hm)
    h = torch.stack([e[n - k - 1] - e[n - k] for k in range(n)])
    return torch.where(wet, h, o.h_src), wet


def _ppm_edges(h, act):
    m = act.to(F64)
    west = lambda a, fill: torch.cat([fill(a), a[..., :-1]], -1)                                       # noqa: E731
    east = lambda a, fill: torch.cat([a[..., 1:], fill(a)], -1)                                        # noqa: E731
    mw = west(m, lambda a: torch.zeros_like(a[..., :1]))
    me = east(m, lambda a: torch.zeros_like(a[..., -1:]))
    hm = mw * west(h, lambda a: a[..., :1]) + (1 - mw) * h
    hp = me * east(h, lambda a: a[..., -1:]) + (1 - me) * h
    s = 0.5 * (hp - hm)
    dmx = torch.maximum(torch.maximum(hp, hm), h) - h
    dmn = h - torch.minimum(torch.minimum(hp, hm), h)
    s = torch.sign(s) * torch.minimum(s.abs(), 2 * torch.minimum(dmx, dmn))
    s = torch.where(mw * me * m > 0, s, 0.0)
    hw = 0.5 * (hm + h) + (west(s, lambda a: torch.zeros_like(a[..., :1])) - s) / 6
    he = 0.5 * (hp + h) + (s - east(s, lambda a: torch.zeros_like(a[..., -1:]))) / 6
    curv, dh = 3 * ((hw + he) - 2 * h), he - hw
    inside = (curv > 0) & (dh.abs() < curv)
    num, den = 12 * curv * (h - 2e-10), curv * curv + 3 * dh * dh
    sc = torch.where(inside & (num < den), num / torch.where(den > 0, den, 1.0), 1.0)
    sc = torch.where(inside & (h <= 2e-10), 0.0, sc)
    return h + sc * (hw - h), h + sc * (he - h)


def _ppm_transport(h, ut, L, Qb, qe, qw, act, dt: float, dx):
    """Layer fluxes with PPM thickness whose sum is the barotropic transport (a velocity shift per face column)."""
    n, ny, nx = h.shape
    iw, ie = torch.arange(-1, nx, device="cuda").clamp(min=0), torch.arange(nx + 1, device="cuda").clamp(max=nx - 1)
    hw, he = _ppm_edges(h, act)
    open_ = act[:, iw] & act[:, ie]
    dxw, dxe = dx[:, iw], dx[:, ie]

    def flux(u):
        pos = u >= 0
        pick = lambda a, b: torch.where(pos, a, b)                                                    # noqa: E731
        hu = pick(h[..., iw], h[..., ie])
        edge, far = pick(he[..., iw], hw[..., ie]), pick(hw[..., iw], he[..., ie])
        q = pick(qe, qw)
        c = (u.abs() * dt / torch.where(pos, dxw, dxe)).clamp(max=1)
        curv, dh = (edge + far) - 2 * hu, far - edge
        mean = edge + c * (0.5 * dh + curv * (c - 1.5))
        marg = edge + c * (dh + 3 * curv * (c - 1))
        cut = q < hu
        mean, marg = torch.where(cut, torch.minimum(mean, q), mean), torch.where(cut, torch.minimum(marg, q), marg)
        return torch.where(open_, L * u * mean.clamp(min=0), 0.0), torch.where(open_, L * marg.clamp(min=0), 0.0)

    hi = torch.minimum(0.5 * dxw / dt, (0.5 * dxw / dt - ut).amin(0)).clamp(min=0)
    lo = torch.maximum(-0.5 * dxe / dt, (-(0.5 * dxe / dt + ut)).amax(0)).clamp(max=0)
    du = torch.zeros_like(hi)
    F, dF = flux(ut)
    err, ds = F.sum(0) - Qb, dF.sum(0)
    for _ in range(20):
        hi, lo = torch.where(err > 0, du, hi), torch.where(err < 0, du, lo)
        step = torch.where(ds > 0, -err / torch.where(ds > 0, ds, 1.0), 0.0)
        new = du + step
        new = torch.where((step > 0) & (new >= hi), 0.5 * (du + hi), new)
        du = torch.where((step < 0) & (new <= lo), 0.5 * (du + lo), new)
        F, dF = flux(ut + du)
        err, ds = F.sum(0) - Qb, dF.sum(0)
        if bool((err.abs() <= 1e-12 * Qb.abs().clamp(min=1)).all()):
            break
    R = Qb - F.sum(0)
    te, tw = qe.sum(0), qw.sum(0)
    use_e = torch.where(R >= 0, te > 0, tw <= 0)
    tot = torch.where(use_e, te, tw)
    return torch.where(open_, F + R * torch.where(use_e, qe, qw) / torch.where(tot > 0, tot, 1.0), 0.0)


def _layer_transport(o) -> dict:
    def velocity(un, uo, wet, w, L, D):
        uo = torch.where(wet, uo, 0.0)
        x = 0.5 * un + 0.5 * uo + (0.6 - 0.5) * ((w * un).sum(0) - (w * uo).sum(0))
        return x, L * D * (w * x).sum(0)

    ux, bx = velocity(o.u1, o.u0, o.wet_u, o.wu, o.Lu, o.Du)
    uy, by = velocity(o.v1, o.v0, o.wet_v, o.wv, o.Lv, o.Dv)
    Qx = _ppm_transport(o.h, ux, o.Lu, bx, o.qe, o.qw, o.wet, o.dt, o.dx)
    Qy = _tr(_ppm_transport(_tr(o.h), _tr(uy), o.Lv.T, by.T, o.qn, o.qs, o.wet.T, o.dt, o.dy.T)).contiguous()
    area = torch.where(o.wet, o.area, 0.0)
    out = torch.clamp(Qx[..., 1:], min=0) - torch.clamp(Qx[..., :-1], max=0) + torch.clamp(Qy[:, 1:], min=0) \
        - torch.clamp(Qy[:, :-1], max=0)
    over = o.wet & (out > (o.h - 2e-10).clamp(min=0) * area / o.dt)
    if bool(over.any()):                               # the limiter redistributes: no value of its own here
        return dict(Qx=None, Qy=None, V0=o.h * o.area, V1=None, ok=None, h_dagger=None)
    div = Qx[..., 1:] - Qx[..., :-1] + Qy[:, 1:] - Qy[:, :-1]
    hd = (o.h - o.dt * div / o.area).clamp(min=0)
    V1 = hd * o.area
    return dict(Qx=Qx, Qy=Qy, V0=o.h * o.area, V1=V1, ok=o.wet & (V1 > 0), h_dagger=hd)


def _diffuse(o, kh: float, dt: float):
    outs = []
    for t in range(o.C.shape[0]):
        Tw = o.Tw[t]
        fx, fy = torch.zeros_like(o.Qx), torch.zeros_like(o.Qy)
        act = o.wet
        fx[..., 1:-1] = torch.where((act[:, 1:] & act[:, :-1] & o.okx[:, 1:-1]),
                                    -kh * o.cx[:, 1:-1] * torch.minimum(o.h_tgt[..., :-1], o.h_tgt[..., 1:])
                                    * (Tw[..., 1:] - Tw[..., :-1]), 0.0)
        fy[:, 1:-1] = torch.where((act[1:] & act[:-1] & o.oky[1:-1]),
                                  -kh * o.cy[1:-1] * torch.minimum(o.h_tgt[:, :-1], o.h_tgt[:, 1:])
                                  * (Tw[:, 1:] - Tw[:, :-1]), 0.0)
        div = fx[..., 1:] - fx[..., :-1] + fy[:, 1:] - fy[:, :-1]
        outs.append(torch.where(o.V0 > 0, o.C[t] - dt * div / torch.where(o.V0 > 0, o.V0, 1.0), o.C[t]))
    return torch.stack(outs)
