"""Spreading and interpolation on grids whose sides are not multiples of the 8-point tile
(tiles of 8 and 7 points) against the stencil sums in numpy: only 7-point tiles (28, 42,
63), one 8-point tile among them and the reverse, odd sides, one uneven side beside whole
ones, the widest stencil that four tiles hold (22 points), one more and sides that cannot
be cut into 7 and 8 (34: the per-blob kernels), blobs on the first and last points, outside
the box and several in one tile.  A grid point or velocity is a sum of at most 60 or 22^3
products in FP64: 1e-13 norm-wise; FP32 weights, products and sums as the rest of the
suite, 1e-6."""
import math

import numpy as np
import pytest

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu

DX, NB = 0.45, 60


def _stencils(Y, W):
    """First points (n, 3) and weights (n, 3, W)."""
    first = np.trunc(Y / DX).astype(int) - W // 2 + 1
    x = (first[:, :, None] + np.arange(W)) * DX - Y[:, :, None]
    return first, np.exp(-x * x * math.pi / 2.0) / math.sqrt(2.0)


@pytest.mark.parametrize("slip", [0, 1])
@pytest.mark.parametrize("n, W", [((28, 28, 28), 20), ((28, 30, 31), 20), ((36, 42, 63), 20), ((50, 36, 38), 20),
                                  ((32, 40, 30), 22), ((40, 30, 32), 11), ((30, 32, 40), 4), ((57, 58, 42), 22),
                                  ((100, 126, 90), 20), ((62, 46, 44), 23), ((34, 36, 40), 20), ((64, 30, 34), 12)])
def test_spread_and_interpolation(gpu, n, W, slip):
    if slip and n[1] % 2:
        n = (n[0], n[1] + 1, n[2])
    rng = np.random.default_rng(sum(n) + W)
    L = DX * np.array(n)
    Y = rng.uniform(-0.3, 1.3, (NB, 3)) * L
    Y[:3] = [[0, 0, 0], L - 1e-9, [0, 0.5 * L[1], L[2] - 1e-9]]
    Y[40:] = 0.5 * L + 2.0 * rng.uniform(-1, 1, (NB - 40, 3))
    F = rng.standard_normal((NB, 3))
    g = Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=W, dx=DX, num_bodies=NB, blobs_per_body=1,
                                      ncells=3, precision=1, slip_channel=slip), [0, 0, 0])
    g.set_up_gaussians(Y.ravel())
    first, w = _stencils(Y, W)
    ix = [(first[:, d, None] + np.arange(W)) % n[d] for d in range(3)]
    at = lambda b: np.ix_(ix[0][b], ix[1][b], ix[2][b])
    prod = lambda b: w[b, 0][:, None, None] * w[b, 1][None, :, None] * w[b, 2][None, None, :]
    ref = np.zeros((3,) + tuple(n))
    for b in range(NB):
        for c in range(3):
            ref[c][at(b)] += F[b, c] * prod(b)
    if slip:
        h = n[1] // 2
        ref[1][:, 0] = ref[1][:, h] = 0
        for c, sign in ((0, 1), (1, -1), (2, 1)):
            ref[c][:, h + 1:] = sign * ref[c][:, h - 1:0:-1]
    g.spread(F.ravel(), 0)
    got = [np.asarray(u).reshape(n[0], n[1], -1)[:, :, :n[2]] for u in g.get_velocity_field(0)]
    for c in range(3):
        assert rel_err(got[c], ref[c]) < 1e-13
    V = np.zeros((NB, 3))
    for b in range(NB):
        p = prod(b)
        if slip:
            p = p * (ix[1][b] < n[1] // 2)[None, :, None]
        V[b] = [DX ** 3 * np.sum(ref[c][at(b)] * p) for c in range(3)]
    assert rel_err(g.interp(0), V.ravel()) < 1e-13
    g.spread(F.ravel(), 1)
    assert rel_err(g.interp(1), V.ravel()) < 1e-6


@pytest.mark.parametrize("nb", [1, 31, 32, 33, 63, 64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("n", [(32, 32, 32), (36, 30, 45)])
def test_long_tile_lists(gpu, n, nb):
    """Tile lists of as many blobs as a lane's one, two, four or eight entries hold, and one
    more: the sums against numpy, and the same bits from a second set-up
    (the lists are filled in any order).  Tolerance as above."""
    W = 20
    rng = np.random.default_rng(nb)
    Y = DX * (np.array(n) / 2 + rng.uniform(-0.9, 0.9, (nb, 3)))
    F = rng.standard_normal((nb, 3))
    g = Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=W, dx=DX, num_bodies=nb, blobs_per_body=1,
                                      ncells=3, precision=0), [0, 0, 0])
    first, w = _stencils(Y, W)
    ref = np.zeros((3,) + tuple(n))
    for b in range(nb):
        at = np.ix_(*[(first[b, d] + np.arange(W)) % n[d] for d in range(3)])
        p = w[b, 0][:, None, None] * w[b, 1][None, :, None] * w[b, 2][None, None, :]
        for c in range(3):
            ref[c][at] += F[b, c] * p
    runs = []
    for _ in range(2):
        g.set_up_gaussians(Y.ravel())
        g.spread(F.ravel(), 0)
        runs.append([np.asarray(u).reshape(n[0], n[1], -1)[:, :, :n[2]].copy() for u in g.get_velocity_field(0)])
    for c in range(3):
        assert rel_err(runs[0][c], ref[c]) < 1e-13
        assert np.array_equal(runs[0][c], runs[1][c])
