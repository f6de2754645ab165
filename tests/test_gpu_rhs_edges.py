"""The single evaluation of the faces and the RHS on ragged grids and masks, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import pyocean_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _adv(mod, scheme, open_):
    return mod.TracerAdvection(scheme=scheme, time="ssprk3", dt=1.0, ob=mod.OpenEdges(open_))


@pytest.mark.parametrize("scheme", ["weno5", "weno5js"])
@pytest.mark.parametrize("grid", [(1, 1, 1, 1), (2, 2, 3, 5), (1, 3, 6, 7), (3, 5, 8, 32), (2, 6, 11, 38), (1, 9, 25, 70)],
                         ids=lambda g: "x".join(map(str, g)))
def test_single_evaluation(grid, scheme):
    nt, n, ny, nx = grid
    rng = np.random.default_rng(sum(grid))
    c = rng.normal(10.0, 1.0, grid)
    Qx, Qy = rng.normal(0, 1, (n, ny, nx + 1)), rng.normal(0, 1, (n, ny + 1, nx))
    Fz = rng.normal(0, 1, (n + 1, ny, nx))
    for q in (Qx, Qy, Fz):
        q *= rng.random(q.shape) > 0.2                                 # faces without transport
    Fz[0] = Fz[-1] = 0.0
    ok = rng.random((n, ny, nx)) > 0.2
    for open_, infl in (((), None), (("west", "north"), c + 1.0)):
        gpu, ref = _adv(P, scheme, open_), _adv(O, scheme, open_)
        for z, zr in ((Fz, Fz), (None, np.zeros_like(Fz))):            # the oracle takes no transport as zeros
            np.testing.assert_array_equal(gpu.rhs(c, Qx, Qy, z, ok, inflow=infl), ref.rhs(c, Qx, Qy, zr, ok, inflow=infl))
        for a, b in zip(gpu.faces_h(c, Qx, Qy, ok, inflow=infl), ref.faces_h(c, Qx, Qy, ok, inflow=infl)):
            np.testing.assert_array_equal(a, b)
