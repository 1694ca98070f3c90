"""The FP64 fluctuating field of slender boxes, on either side of the rule that gives them to
cuFFT's transform (from 140 points along x, fewer than 222 CTAs of the x pass), against the
same draws in FP32 with cuFFT's transform: norm-wise 2e-6, as the other test of the field.
And its time in a box of 512 x 16 x 8 points against the FP32 field's there."""
import numpy as np
import pytest
import torch

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu


def _context(n, prec, slip=0):
    return Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=4, dx=1.0, num_bodies=2, blobs_per_body=1,
                                         ncells=3, precision=prec, algorithm=2, slip_channel=slip), [0, 0, 0],
                      stream=torch.cuda.current_stream())


@pytest.mark.parametrize("slip", [0, 1])
@pytest.mark.parametrize("n", [(140, 36, 48), (140, 40, 48), (200, 36, 48), (200, 40, 48), (256, 36, 24), (256, 40, 24),
                               (288, 54, 16), (288, 56, 16), (384, 72, 12), (384, 80, 12), (512, 36, 24), (512, 40, 24),
                               (512, 42, 42), (320, 100, 90), (128, 8, 8)])
def test_field(gpu, n, slip):
    fields = []
    for prec in (0, 1):
        g = _context(n, prec, slip)
        g.produce_random_velocity_field(11, 7)
        fields.append([np.asarray(u).reshape(n[0], n[1], -1)[:, :, :n[2]] for u in g.get_velocity_field(1)])
    for a, b in zip(*fields):
        assert np.any(a) and rel_err(b, a) < 2e-6


def test_time(gpu):
    us = []
    for prec in (0, 1):
        g = _context((512, 16, 8), prec)
        best = 1e30
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                g.produce_random_velocity_field(1, 2)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 50.0)
        us.append(best)
    print("512 x 16 x 8: FP64 %.1f us, FP32 %.1f us" % tuple(us))
    assert us[0] < 1.6 * us[1]
