"""The Stokes solve on the packed half spectrum (FP64 solve variant 1, FP32 variant 2; the
default where all three lengths are supported) on the shapes where it can go wrong: the
smallest lengths (tiles padded beyond H/2 columns, fewer columns than a tile), lengths that
are not whole numbers of tile columns, planes by one CTA and by separate passes, both tile
shapes (256 points along x and more), the longest lengths, and narrow Gaussians (ngauss 4,
sigma = 0.56 dx), whose spectrum is far from zero in the Nyquist rows and planes where the
projection is symmetrised.  The whole velocity field is compared with the oracle's: norm-wise
1e-12 in FP64 (a few hundred roundings), 1e-6 in FP32 as the rest of the suite."""
import numpy as np
import pytest

from tests.conftest import rel_err
from tests.oracle_lib import Oracle
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu


def _params(n, nb, **kw):
    return FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=4, dx=1.0, num_bodies=nb, blobs_per_body=1, ncells=3,
                              precision=1, **kw)


def _against_oracle(n):
    nb = 30
    rng = np.random.default_rng(sum(n))
    Y = (rng.uniform(0, 1, (nb, 3)) * np.array(n)).ravel()
    F = rng.standard_normal(3 * nb)
    p = _params(n, nb)
    g, o = Suspension(p, [0, 0, 0]), Oracle(p.copy(precision=0), [0, 0, 0])
    for s in (g, o):
        s.set_up_gaussians(Y)
        s.set_up_force_distribution(F)
        s.produce_deterministic_velocity_field()
    ug = g.get_velocity_field(0)
    for c in range(3):
        a, b = (np.asarray(u).reshape(n[0], n[1], -1)[:, :, :n[2]] for u in (ug[c], o.get_grid(3 + c)))
        assert rel_err(a, b) < 1e-12, c
    Vo = o.calculate_deterministic_blob_velocities()
    g.spread(F, 1)
    g.stokes_solve(1)
    assert rel_err(g.interp(1), Vo) < 1e-6
    return g


@pytest.mark.parametrize("n", [(8, 8, 8), (12, 8, 12), (8, 12, 16), (16, 8, 12), (24, 16, 8), (24, 24, 24),
                               (48, 12, 16), (64, 32, 24), (96, 8, 48), (192, 16, 12), (256, 12, 8), (256, 16, 96),
                               (8, 384, 16), (8, 16, 384), (12, 512, 512), (384, 8, 8), (384, 16, 24), (512, 8, 12),
                               (512, 12, 16), (16, 48, 48), (8, 96, 96)])
def test_velocity_field(gpu, n):
    assert _against_oracle(n).get_variants()[3] == 2


@pytest.mark.parametrize("n", [36, 40, 42, 50, 54, 56, 60, 70, 72, 80, 84, 90, 98, 100, 108, 112, 120, 126, 140, 144,
                               150, 160, 162, 168, 180, 196, 200, 210, 216, 224, 240, 252, 270, 280, 288, 300, 320,
                               400, 480])
def test_velocity_field_lengths(gpu, n):
    """The lengths with 5, 7 or 9 among their register sizes, along each direction and, up
    to 96 points, as planes by one CTA; half of them odd along z (no column H/2), so are
    those of the 126 by 90 box.  Tolerances as above."""
    shapes = [(8, n, 8), (8, 8, n)]
    if n % (8 if n >= 256 else 4) == 0:
        shapes += [(n, 8, 12), (n, 12, 90)]
    if n <= 96:
        shapes.append((8, n, n))
    if n in (90, 126):
        shapes.append((256, 126, 90) if n == 90 else (100, 126, 90))
    for shape in shapes:
        _against_oracle(shape)


@pytest.mark.parametrize("slip", [0, 1])
@pytest.mark.parametrize("n", [(8, 8, 8), (16, 24, 12), (40, 42, 90), (100, 16, 42), (24, 16, 16), (64, 48, 32), (256, 8, 16), (384, 12, 8)])
def test_fluctuating_field(gpu, n, slip):
    """The FP64 fluctuating field, drawn inside the x pass of the packed spectrum, against
    the same draws in the whole half spectrum with cuFFT's 3D transform, which the FP32
    field of a mixed-precision context takes: norm-wise 2e-6 (FP32 amplitudes and
    transform), with the slip channel's image-symmetric stress and without."""
    nb = 2
    fields = []
    for prec in (0, 1):
        g = Suspension(_params(n, nb, slip_channel=slip).copy(precision=prec), [0, 0, 0])
        g.produce_random_velocity_field(11, 7)
        fields.append([np.asarray(u).reshape(n[0], n[1], -1)[:, :, :n[2]] for u in g.get_velocity_field(1)])
    for a, b in zip(*fields):
        assert np.any(a) and rel_err(b, a) < 2e-6
