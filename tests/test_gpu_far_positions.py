"""Blobs at infinite positions, or more grid spacings away than an int holds, among ordinary
ones: they meet no tile (their weights are zero), so they spread nothing and their velocity is
zero, and the others get the velocities they have without them (FP64 1e-13, FP32 1e-6: the
tile lists hold the same blobs in the same order).  Every direction and sign, two and three
directions at once (the product of the counts of tiles is then positive though each is
negative), on whole and uneven tiles and on a grid that is not cut into tiles."""
import numpy as np
import pytest

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu

DX = 0.45
FAR = [(np.inf, 3, 4), (3, np.inf, 4), (3, 4, -np.inf), (np.inf, np.inf, 4), (-np.inf, 3, np.inf), (5, 1e300, -1e300),
       (np.inf, np.inf, np.inf), (-np.inf, -np.inf, -np.inf), (1e12, 1e12, 5.0)]


def _velocities(n, W, Y, F):
    g = Suspension(FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=W, dx=DX, num_bodies=len(Y), blobs_per_body=1,
                                      ncells=3, precision=1), [0, 0, 0])
    g.set_up_gaussians(Y.ravel())
    out = []
    for P in (0, 1):
        g.spread(F.ravel(), P)
        g.stokes_solve(P)
        for v in (0, 1, 2):
            w = g.get_variants()
            w[4 + P] = v
            g.set_variants(w)
            out.append((P, g.interp(P).reshape(-1, 3).copy()))
    return out


@pytest.mark.parametrize("W", [20, 11, 2])
@pytest.mark.parametrize("n", [(32, 32, 32), (36, 30, 45), (28, 42, 30), (34, 36, 40)])
def test_far_blobs(gpu, n, W):
    rng = np.random.default_rng(W)
    near = rng.uniform(0, 1, (25, 3)) * DX * np.array(n)
    F = rng.standard_normal((len(near) + len(FAR), 3))
    ref = _velocities(n, W, near, F[:len(near)])
    got = _velocities(n, W, np.concatenate([near, np.array(FAR, dtype=float)]), F)
    for (P, a), (_, b) in zip(ref, got):
        assert np.all(np.isfinite(b)) and np.any(a)
        assert not np.any(b[len(near):])
        assert rel_err(b[:len(near)], a) < (1e-13 if P == 0 else 1e-6)
