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


def _flow(seed, n, ny, nx, kind):
    rng = np.random.default_rng(seed)
    H = rng.uniform(20.0, 400.0, (ny, nx))
    act = rng.random((ny, nx)) > 0.08
    h = np.where(act[None], H / n * rng.uniform(0.5, 1.5, (n, ny, nx)), np.nan)
    q_e, q_w = O.face_transport_thickness(h, np.nan_to_num(h).sum(0), act, True)
    L, dx = rng.uniform(1800.0, 2200.0, (ny, nx + 1)), rng.uniform(1800.0, 2200.0, (ny, nx))
    noise = rng.normal(0.0, 0.3, (n, ny, nx + 1))
    if kind == "coherent":                                     # columns of one direction: a few steps
        ut = rng.choice([-1.0, 1.0], (ny, nx + 1)) * (0.1 + 0.03 * noise)
        off = rng.uniform(0.8, 1.2, L.shape)
    elif kind == "strong":                                     # one direction, corrections of the size of the flow
        ut = 0.4 + 0.1 * noise
        off = rng.uniform(-2.0, 4.0, L.shape)
    else:                                                      # a coherent part and a part that never settles
        ut, off = 0.1 + 0.03 * noise, rng.uniform(0.8, 1.2, L.shape)
        ut[:, -1:] = noise[:, -1:]
    Q = (L[None] * ut * 0.5 * (q_e + q_w)).sum(0) * off
    return h, ut, L, Q, q_e, q_w, act, dx


@pytest.mark.parametrize("max_iter", [2, 5, 20, 40])
@pytest.mark.parametrize("kind", ["coherent", "strong", "part"])
@pytest.mark.parametrize("n,ny,nx", [(5, 3, 40), (32, 6, 50), (50, 5, 61), (75, 3, 33), (81, 2, 40)])
def test_iterations_that_settle_at_different_steps(n, ny, nx, kind, max_iter):
    case = _flow(n, n, ny, nx, kind)
    got = P.ppm_transport_x(*case[:-1], 300.0, case[-1], max_iter)
    np.testing.assert_array_equal(got, O.ppm_transport_x(*case[:-1], 300.0, case[-1], max_iter))


# The settling step of a large grid of deep columns, most of which stop early: one direction (settles everywhere), a part
# that never settles, and faces whose sums round as coarsely as the tolerance, which converge and then have not.
def _large(kind):
    n, ny, nx = 53, 114, 540
    h = np.tile(np.random.default_rng(10 ** 6).uniform(0.5, 1.5, (n, 1, 12)) * 5.0, (1, ny, nx // 12))
    act, q = np.ones((ny, nx), bool), np.full((n, ny, nx + 1), 1e3)
    L, dx = np.full((ny, nx + 1), 2000.0), np.full((ny, nx), 2000.0)
    ut = np.full((n, ny, nx + 1), 0.1)
    if kind != "again":
        ut *= np.random.default_rng(1).uniform(0.7, 1.3, ut.shape)
    off = np.random.default_rng(2).uniform(0.9, 1.1, L.shape) if kind != "again" else 1.0
    Q = np.zeros(L.shape)
    for k in range(n):
        Q += L * ut[k] * 5.0
    Q *= off
    blocks = (ny * (nx + 1) + 31) // 32
    part = (blocks + 63) // 64                                  # the CTAs take 64 parts of the grid side by side

    def place(seed, block):
        """A face of noise in this block, with the column's neighbours as every twelfth face has them."""
        o = next(o for o in range(block * 32, block * 32 + 32) if o % (nx + 1) % 12 == 6 and 0 < o % (nx + 1) < nx)
        rng = np.random.default_rng(seed)
        ut[:, o // (nx + 1), o % (nx + 1)] = rng.normal(0.0, 0.3, n)
        Q[o // (nx + 1), o % (nx + 1)] = rng.uniform(-100.0, 100.0)

    if kind == "again":
        for i, seed in enumerate((494, 501, 701, 841, 1472, 1500)):      # converged after step 2, not after step 3
            place(seed, (5 + 8 * i) * part + 2 * part // 3)
        for i, seed in enumerate((192, 610, 1378, 2246)):                # converged after step 3, not after step 4
            place(seed, (7 + 8 * i) * part + part - 1)
    elif kind == "never":
        place(19, 40 * part + part - 1)                          # rounds more coarsely than its tolerance
    return h, ut, L, Q, q, q, act, dx


@pytest.mark.parametrize("max_iter", [3, 20])
@pytest.mark.parametrize("kind", ["settles", "never", "again"])
def test_columns_that_stop_early(kind, max_iter):
    import torch

    from pyocean_b200 import _lib
    L_ = _lib.lib()
    case = _large(kind)
    n, ny, nf = case[1].shape
    h, ut, L, Q, q_e, q_w, act, dx = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in case)
    nbytes = L_.pocean_ppm_transport_workspace_bytes(n, ny, nf - 1, max_iter)
    ws, out = torch.empty(nbytes, dtype=torch.uint8, device="cuda"), torch.empty_like(ut)
    _lib.check(L_.pocean_ppm_transport_f64(
        h.data_ptr(), ut.data_ptr(), L.data_ptr(), Q.data_ptr(), q_e.data_ptr(), q_w.data_ptr(), act.data_ptr(),
        dx.data_ptr(), n, ny, nf - 1, 300.0, max_iter, out.data_ptr(), ws.data_ptr(), nbytes,
        torch.cuda.current_stream().cuda_stream), "ppm")
    marks = ws[-((4 * (max_iter + 1) + 255) // 256 * 256):].view(torch.int32)[:max_iter + 1].tolist()
    if max_iter == 20:                                          # the paths meant are the ones that ran
        assert (marks[19] == 1) == (kind == "never") and (marks[20] == -1) == (kind == "again"), marks
    np.testing.assert_array_equal(out.cpu().numpy(), O.ppm_transport_x(*case[:-1], 300.0, case[-1], max_iter))
