"""The layer state's single pass against the passes it stands for, and the plane transposes, at tile edges, bit for bit."""
from __future__ import annotations

import pytest
import torch

from pyocean_b200 import _lib
from pyocean_b200.producers import _swap

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (3, 8, 32), (2, 9, 33), (5, 65, 7), (1, 31, 300), (40, 2, 1)]


def _bits(t):
    return t.view(torch.int64)


@pytest.mark.parametrize("n,ny,nx", SHAPES)
def test_one_pass_equals_the_separate_passes(n, ny, nx):
    g = torch.Generator(device="cuda").manual_seed(100 * n + ny)
    f = dict(generator=g, dtype=torch.float64, device="cuda")
    h = torch.rand((n, ny, nx), **f) * 10.0
    Qx, Qy = torch.randn((n, ny, nx + 1), **f), torch.randn((n, ny + 1, nx), **f)
    area = torch.rand((ny, nx), **f) * 100.0
    act = (torch.rand((ny, nx), **f) < 0.8).to(torch.uint8)
    area[act == 0] = 0.0
    h.view(-1)[::7] = 0.0                          # emptied layers: negative h-dagger
    if h.numel() > 8:
        h.view(-1)[3] = float("nan")
    L, st, p = _lib.lib(), torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()
    div, hd, V0, V1 = (torch.empty_like(h) for _ in range(4))
    ok = torch.empty((n, ny, nx), dtype=torch.uint8, device="cuda")
    bad = torch.empty(2, dtype=torch.int64, device="cuda")
    for dt, tol in ((0.5, 1e-9), (3.0, 0.01)):
        assert L.pocean_flux_divergence_f64(p(Qx), p(Qy), n, ny, nx, p(div), st) == 0
        assert L.pocean_lagrangian_thickness_f64(p(h), p(div), p(area), n, ny, nx, dt, tol, p(hd), p(bad), st) == 0
        assert L.pocean_layer_volumes_f64(p(h), p(area), p(act), n, ny, nx, p(V0), None, st) == 0
        assert L.pocean_layer_volumes_f64(p(hd), p(area), p(act), n, ny, nx, p(V1), p(ok), st) == 0
        got = [torch.full_like(h, -1.0) for _ in range(3)]
        okg = torch.full_like(ok, 9)
        assert L.pocean_layer_state_f64(p(h), p(Qx), p(Qy), p(area), p(act), n, ny, nx, dt, tol, p(got[0]), p(got[1]),
                                        p(got[2]), p(okg), p(bad) + 8, st) == 0
        for a, b in zip(got, (hd, V0, V1)):
            assert torch.equal(_bits(a), _bits(b))
        assert torch.equal(okg, ok)
        assert int(bad[0]) == int(bad[1])


@pytest.mark.parametrize("n,ny,nx", SHAPES)
def test_transpose(n, ny, nx):
    t = torch.arange(n * ny * nx, dtype=torch.float64, device="cuda").view(n, ny, nx)
    assert torch.equal(_swap(t), t.transpose(-1, -2).contiguous())
    assert torch.equal(_swap(t[0]), t[0].t().contiguous())
    assert torch.equal(_swap(t[:, :, ::2]), t[:, :, ::2].transpose(-1, -2).contiguous())      # a strided view
