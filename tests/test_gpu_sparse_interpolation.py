"""FP64 tile interpolation where most tiles hold no blob: those are not read.  The velocities
against the 64-thread kernel (variant 0) to FP64 summation order, with blobs in the first and
last tile, several rounds of one tile beside empty ones, and in the slip channel; and the time
of a few blobs in a 256^3 grid against that kernel, whose CTAs of empty tiles return at once
(reading all of the 403 MB takes 2.5 times as long)."""
import numpy as np
import pytest
import torch

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu

DX = 0.45


def _context(n, Y, F, slip=0):
    g = Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=12, dx=DX, num_bodies=len(Y), blobs_per_body=1,
                                      ncells=3, slip_channel=slip), [0, 0, 0], stream=torch.cuda.current_stream())
    g.set_up_gaussians(Y.ravel())
    g.spread(F.ravel(), 0)
    g.stokes_solve(0)  # a velocity at every point
    return g


def _variant(g, v):
    w = g.get_variants()
    w[4] = v
    g.set_variants(w)


@pytest.mark.parametrize("slip", [0, 1])
@pytest.mark.parametrize("n", [(160, 128, 96), (60, 124, 130)])
@pytest.mark.parametrize("nb, crowd", [(1, 0), (2, 0), (3, 40), (5, 17), (40, 100)])
def test_velocities(gpu, n, nb, crowd, slip):
    rng = np.random.default_rng(nb + crowd)
    L = DX * np.array(n)
    Y = rng.uniform(0, 1, (nb + crowd, 3)) * L
    Y[0] = 1e-9
    Y[nb - 1] = L - 1e-9
    Y[nb:] = 0.4 * L + rng.uniform(0, 2, (crowd, 3))
    g = _context(n, Y, rng.standard_normal((nb + crowd, 3)), slip)
    _variant(g, 0)
    ref = g.interp(0).copy()
    _variant(g, 1)
    assert np.any(ref) and rel_err(g.interp(0), ref) < 1e-13


@pytest.mark.parametrize("nb", [1, 66])
def test_time_of_few_blobs(gpu, nb):
    n = (256, 256, 256)
    rng = np.random.default_rng(nb)
    g = _context(n, rng.uniform(0, 1, (nb, 3)) * DX * np.array(n), rng.standard_normal((nb, 3)))
    V = torch.empty(3 * nb, dtype=torch.float64, device="cuda")
    us = {}
    for v in (0, 1, 0, 1):
        _variant(g, v)
        for _ in range(3):
            g.interp(0, out=V)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(20):
            g.interp(0, out=V)
        b.record()
        torch.cuda.synchronize()
        us[v] = min(us.get(v, 1e30), a.elapsed_time(b) * 50.0)
    print("%d blobs: variant 0 %.1f us, variant 1 %.1f us" % (nb, us[0], us[1]))
    assert us[1] < 1.5 * us[0]
