"""The PPM layer transport around its layer counts and stopping rules, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from pyocean_b200 import producers as P

pytestmark = pytest.mark.gpu


def _faces(seed, n, ny, nx, flow):
    rng = np.random.default_rng(seed)
    H = rng.uniform(20.0, 400.0, (ny, nx))
    act = rng.random((ny, nx)) > 0.1
    h = np.stack([H / n * rng.uniform(0.5, 1.5, (ny, nx)) for _ in range(n)])
    h[0, :, : nx // 4] = 0.0
    h = np.where(act[None], h, np.nan)
    q_e, q_w = O.face_transport_thickness(h, np.nan_to_num(h).sum(0), act, True)
    L, dx = rng.uniform(1800.0, 2200.0, (ny, nx + 1)), rng.uniform(1800.0, 2200.0, (ny, nx))
    if flow == "rest":                                    # converged from the start
        ut = np.zeros((n, ny, nx + 1))
        return h, ut, L, np.zeros((ny, nx + 1)), q_e, q_w, act, dx
    ut = rng.normal(0.0, 0.3, (n, ny, nx + 1))
    if flow == "coherent":                                # one sign, small transports: converges in a few steps
        ut = 1e-6 * (1.0 + 0.1 * ut)
    ut[:, :, ::6] = 0.0
    ut[:, 0, ::5] = -0.0
    Q = (L[None] * ut * 0.5 * (q_e + q_w)).sum(0) * rng.uniform(0.9, 1.1, L.shape)
    return h, ut, L, Q, q_e, q_w, act, dx


@pytest.mark.parametrize("max_iter", [0, 1, 2, 20])
@pytest.mark.parametrize("flow", ["noise", "coherent", "rest"])
@pytest.mark.parametrize("n,ny,nx", [(1, 1, 1), (3, 2, 31), (32, 3, 33), (33, 2, 40), (56, 2, 20), (57, 3, 21), (80, 1, 35),
                                     (81, 2, 17)])
def test_ppm_transport_around_the_layer_counts(n, ny, nx, flow, max_iter):
    h, ut, L, Q, q_e, q_w, act, dx = _faces(n + ny, n, ny, nx, flow)
    got = P.ppm_transport_x(h, ut, L, Q, q_e, q_w, act, 300.0, dx, max_iter)
    np.testing.assert_array_equal(got, O.ppm_transport_x(h, ut, L, Q, q_e, q_w, act, 300.0, dx, max_iter))


@pytest.mark.parametrize("what", ["inf", "nan", "huge", "tiny", "width"])
def test_faces_outside_the_short_quotients(what):
    h, ut, L, Q, q_e, q_w, act, dx = _faces(5, 12, 4, 70, "noise")
    if what == "inf":
        ut[3, 1, 20], ut[4, 2, 40] = np.inf, -np.inf
    elif what == "nan":
        ut[3, 1, 20] = np.nan
    elif what == "huge":
        ut[3, 1, 20] = 1e200
    elif what == "tiny":
        ut[:, 1, 20:30] *= 1e-200
        Q[1, 20:30] *= 1e-200
    else:
        dx[1, 20], dx[2, 30] = 0.0, 1e-150
    with np.errstate(all="ignore"):
        got = P.ppm_transport_x(h, ut, L, Q, q_e, q_w, act, 300.0, dx)
        np.testing.assert_array_equal(got, O.ppm_transport_x(h, ut, L, Q, q_e, q_w, act, 300.0, dx))


@pytest.mark.parametrize("ny,nx", [(1, 1), (2, 2), (3, 29), (2, 30), (1, 31), (2, 60), (2, 61), (1, 121), (3, 150)])
def test_edges_around_the_warp_tiles(ny, nx):
    rng = np.random.default_rng(nx)
    h = rng.uniform(0.0, 3.0, (3, ny, nx)) * (rng.random((3, ny, nx)) > 0.2)
    h[0, 0, 0] = np.nan
    act = rng.random((ny, nx)) > 0.15
    for got, ref in zip(P.ppm_edges_x(h, act), O.ppm_edges_x(h, act)):
        np.testing.assert_array_equal(got, ref)
