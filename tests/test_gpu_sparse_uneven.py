"""Few blobs on uneven grids: where the per-blob kernels take over from the tiles, at the edges
of the rules (one blob below and at each).  Spreading by tiles on grids beyond the L2 from
one blob per 32 tiles on in FP64 (186^3: 13,824 tiles) and 14 in FP32 (210^3: 19,683);
interpolation from one per 16 in FP64 (126^3: 4096) and from 600 and one per 12 in FP32 (62^3: 512).
The force grid and the velocities against the stencil sums in numpy: sums of at most a few
dozen, and 20^3, products, 1e-13 in FP64 and 1e-6 in FP32 norm-wise as the other tests of
uneven tiles.  And the time of a sparse product on a 250^3 grid against the 256^3 grid, which
has 7% more points and whole tiles."""
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
    return Suspension(FcmParams.defaults(nx=n, ny=n, nz=n, ngauss=W, dx=DX, num_bodies=nb, blobs_per_body=1, ncells=3,
                                         precision=1, **kw), [0, 0, 0], stream=torch.cuda.current_stream())


@pytest.mark.parametrize("n, nb, slip", [(186, 431, 0), (186, 432, 0), (186, 431, 1), (210, 1405, 0), (210, 1406, 0),
                                         (126, 255, 0), (126, 256, 0), (126, 255, 1), (62, 642, 0), (62, 643, 0),
                                         (62, 642, 1)])
def test_edges(gpu, n, nb, slip):
    rng = np.random.default_rng(nb)
    Y = rng.uniform(0, 1, (nb, 3)) * DX * n
    F = rng.standard_normal((nb, 3))
    g = _context(n, nb, slip_channel=slip)
    g.set_up_gaussians(Y.ravel())
    first = np.trunc(Y / DX).astype(int) - W // 2 + 1
    x = (first[:, :, None] + np.arange(W)) * DX - Y[:, :, None]
    w = np.exp(-x * x * math.pi / 2.0) / math.sqrt(2.0)
    ix = (first[:, :, None] + np.arange(W)) % n
    at = [np.ix_(*ix[b]) for b in range(nb)]
    prod = [w[b, 0][:, None, None] * w[b, 1][None, :, None] * w[b, 2][None, None, :] for b in range(nb)]
    ref = np.zeros((3, n, n, n))
    for b in range(nb):
        for c in range(3):
            ref[c][at[b]] += F[b, c] * prod[b]
    h = n // 2
    if slip:
        ref[1][:, 0] = ref[1][:, h] = 0
        for c, sign in ((0, 1), (1, -1), (2, 1)):
            ref[c][:, h + 1:] = sign * ref[c][:, h - 1:0:-1]
    V = np.zeros((nb, 3))
    for b in range(nb):
        p = prod[b] * ((ix[b, 1] < h)[None, :, None] if slip else 1.0)
        V[b] = [DX ** 3 * np.sum(ref[c][at[b]] * p) for c in range(3)]
    for P, tol in ((1, 1e-6), (0, 1e-13)):
        g.spread(F.ravel(), P)
        assert rel_err(g.interp(P), V.ravel()) < tol
    got = g.get_velocity_field(0)
    for c in range(3):
        assert rel_err(np.asarray(got[c]).reshape(n, n, -1)[:, :, :n], ref[c]) < 1e-13


def _product_us(n, nb, P):
    rng = np.random.default_rng(nb)
    g = _context(n, nb)
    Y = torch.from_numpy((rng.uniform(0, 1, (nb, 3)) * DX * n).ravel()).cuda()
    F = torch.from_numpy(rng.standard_normal(3 * nb)).cuda()
    V = torch.empty_like(F)
    best = 1e30
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            g.set_up_gaussians(Y)
            g.spread(F, P)
            g.interp(P, out=V)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 100.0)
    return best


@pytest.mark.parametrize("P", [0, 1])
@pytest.mark.parametrize("nb", [1, 300])
def test_time_of_few_blobs(gpu, nb, P):
    uneven, whole = _product_us(250, nb, P), _product_us(256, nb, P)
    print("%d blobs, precision %d: 250^3 %.0f us, 256^3 %.0f us" % (nb, P, uneven, whole))
    assert uneven < 1.4 * whole
