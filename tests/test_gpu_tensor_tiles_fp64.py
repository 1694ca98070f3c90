"""FP64 spread (variant 0) and interpolation (variant 1) by the FP64 tensor-core tile
kernels at the sizes where their rounds can go wrong: a tile with no blob, one blob,
a partial and a full k-step of four, a partial and a full round of eight (spread) and
sixteen (interpolation), one more than a round, several rounds, and grids of one tile
per CTA and of more tiles than resident CTAs (the pipeline running on across tiles).
The spread grid equals the one-CTA-per-tile FMA kernel's (variant 1) bit for bit: same
products, same order, one rounding per product in either.  The velocities agree with
the other interpolation kernel to FP64 summation order: W^3 = 12^3 terms of one sign
pattern, 1e-13 relative."""
import numpy as np
import pytest

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu


def _context(n, nblobs, slip=0):
    return Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=12, dx=0.5, num_bodies=nblobs,
                                         blobs_per_body=1, ncells=3, slip_channel=slip), [0, 0, 0])


@pytest.mark.parametrize("nblobs", [1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 70])
@pytest.mark.parametrize("n", [(24, 32, 40), (96, 128, 120)])
def test_rounds(gpu, n, nblobs):
    rng = np.random.default_rng(nblobs)
    # every blob inside one tile (its lists hold all of them, ragged lists around it),
    # the last ones on the tile's corner and across the periodic boundary
    Y = (8 + 8 * rng.uniform(0, 1, (nblobs, 3))) * 0.5
    Y[-1] = 4.0
    if nblobs > 4:
        Y[0] = 0.5 * (np.array(n) - 1e-9)
    F = rng.standard_normal(3 * nblobs)
    for slip in (0, 1):
        g = _context(n, nblobs, slip)
        g.set_up_gaussians(Y.ravel())
        out = {}
        for sp in (0, 1):
            v = g.get_variants()
            v[0] = sp
            g.set_variants(v)
            g.spread(F, 0)
            out[sp] = [a.copy() for a in g.get_velocity_field(0)]
        for c in range(3):
            assert np.array_equal(out[0][c], out[1][c])
            assert np.any(out[0][c])
        V = {}
        for ip in (0, 1):
            v = g.get_variants()
            v[4] = ip
            g.set_variants(v)
            V[ip] = g.interp(0).copy()
        assert np.all(np.isfinite(V[1])) and rel_err(V[1], V[0]) < 1e-13
