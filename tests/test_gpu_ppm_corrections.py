"""The PPM layer transport where its correction leaves the ordinary range or settles early, against the oracle bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from pyocean_b200 import producers as P

pytestmark = pytest.mark.gpu


def _hard_quotients(rng, count):
    """Odd B and A < B, both of 53 bits, whose quotient lies next to the middle of two doubles: A 2^54 = N B +- 1, N odd."""
    out = []
    while len(out) < count:
        B = int(rng.integers(1 << 52, 1 << 53)) | 1
        for k in (1, -1):
            A = k * pow(1 << 54, -1, B) % B
            if A >= 1 << 52 and ((A << 54) - k) // B & 1:
                out.append((A, B))
    return np.array(out[:count], dtype=float).T


@pytest.mark.parametrize("max_iter", [1, 2, 3, 20])
def test_tiny_corrections_of_a_column_at_rest(max_iter):
    """Two layers at rest with a tiny outflow to the west: the first step's correction is tiny, and behind it every edge is
    zero (the vanished cell of layer 0; the mean of +-1 in layer 1), so that the next step divides by the Courant number,
    here the hardest quotients to round."""
    rows = 400
    A, B = _hard_quotients(np.random.default_rng(3), rows)
    h = np.zeros((2, rows, 3))
    h[0], h[1] = [1.0, 0.0, 1.0], [-1.0, 1.0, 1.0]
    act = np.ones((rows, 3), bool)
    q = np.full((2, rows, 4), 5.0)
    L, dx = np.full((rows, 4), 2.0), np.repeat(B[:, None] * 2.0 ** -42, 3, axis=1)
    ut, Q = np.zeros((2, rows, 4)), np.zeros((rows, 4))
    Q[:, 1] = -A * 2.0 ** -1060                               # the correction itself: the first slope is 1
    Q[-1, 2] = 1e9                                            # never met: the iteration goes on for every face
    got = P.ppm_transport_x(h, ut, L, Q, q, q, act, 1.0, dx, max_iter)
    ref = O.ppm_transport_x(h, ut, L, Q, q, q, act, 1.0, dx, max_iter)
    np.testing.assert_array_equal(got, ref)
