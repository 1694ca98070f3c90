"""Tile lists longer than a warp's 256 entries: sorted by rank up to 1024, by comparators
beyond, at their edges and with the short lists of the tiles around them.  The sums against
numpy (a grid point adds at most nb products of either sign: nb eps sqrt(nb) = 1e-11 for
2100), and the same bits from a second set-up, which fills the lists in another order; a list
out of order would change them.  A set-up with crowded tiles may cost more than one with the
same blobs apart, but not the square of their number."""
import math

import numpy as np
import pytest
import torch

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu

DX, W = 0.45, 20


def _context(n, nb, **kw):
    return Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=W, dx=DX, num_bodies=nb, blobs_per_body=1,
                                         ncells=3, **kw), [0, 0, 0])


def _crowded(rng, n, nb):
    return DX * (np.array(n) / 2 + rng.uniform(-0.9, 0.9, (nb, 3)))


@pytest.mark.parametrize("nb", [257, 400, 1023, 1024, 1025, 2100])
@pytest.mark.parametrize("n", [(32, 32, 32), (36, 30, 45)])
def test_sums_and_order(gpu, n, nb):
    rng = np.random.default_rng(nb)
    Y = _crowded(rng, n, nb)
    F = rng.standard_normal((nb, 3))
    g = _context(n, nb)
    first = np.trunc(Y / DX).astype(int) - W // 2 + 1
    x = (first[:, :, None] + np.arange(W)) * DX - Y[:, :, None]
    w = np.exp(-x * x * math.pi / 2.0) / math.sqrt(2.0)
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
        assert rel_err(runs[0][c], ref[c]) < 1e-11
        assert np.array_equal(runs[0][c], runs[1][c])


def _set_up_us(g, Y):
    Y = torch.from_numpy(Y.ravel()).cuda()
    best = 1e30
    for _ in range(4):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(5):
            g.set_up_gaussians(Y)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 200.0)
    return best


@pytest.mark.parametrize("n, nb", [((64, 64, 64), 1000), ((62, 62, 62), 1000), ((64, 64, 64), 2000)])
def test_crowded_set_up_time(gpu, n, nb):
    rng = np.random.default_rng(nb)
    g = Suspension(_context(n, nb).p, [0, 0, 0], stream=torch.cuda.current_stream())
    apart = _set_up_us(g, rng.uniform(0, 1, (nb, 3)) * DX * np.array(n))
    crowded = _set_up_us(g, _crowded(rng, n, nb))
    print("%s %d blobs: apart %.0f us, crowded %.0f us" % (n, nb, apart, crowded))
    assert crowded < 30.0 * apart
