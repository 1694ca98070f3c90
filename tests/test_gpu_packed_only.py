"""Grids whose solve is the packed one in every variant (an x length of its own, or FP64 beyond
256 points along x): no cuFFT plan is made for them (its work areas doubled the memory of
the spectrum), injected stress, which needs one, makes it when it comes, and the autotuner
times the one path once and keeps variant 0."""
import gc

import numpy as np
import pytest
import torch

from tests.conftest import rel_err
from timstochrigidbodiessim_b200.fcm import Suspension
from timstochrigidbodiessim_b200.params import FcmParams

pytestmark = pytest.mark.gpu


def _params(n, **kw):
    return FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=8, dx=1.0, num_bodies=10, blobs_per_body=1, ncells=3,
                              **kw)


@pytest.mark.parametrize("n", [(512, 128, 128), (200, 200, 200)])
def test_memory(gpu, n):
    Suspension(_params((64, 64, 64)), [0, 0, 0]).close()
    gc.collect()  # contexts of earlier tests give their memory back now, not in between
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    s = Suspension(_params(n), [0, 0, 0])
    used = free - torch.cuda.mem_get_info()[0]
    arrays = 3 * 3 * 8 * n[0] * n[1] * n[2]  # forces and velocities, spectrum, fluctuating field
    print(n, "%.0f MB, arrays %.0f MB" % (used / 1e6, arrays / 1e6))
    assert arrays < used < 1.2 * arrays
    s.close()


@pytest.mark.parametrize("n", [(384, 16, 24), (40, 48, 50), (64, 48, 32)])
def test_injected_stress(gpu, n):
    """Against the same stress through a context that has cuFFT's plans from the start: the
    two differ in the sides' order only, so does the field (x and z exchanged)."""
    rng = np.random.default_rng(sum(n))
    st = [rng.standard_normal(n) for _ in range(6)]  # xx, yy, zz, xy, xz, yz
    fields = []
    for m, s6 in ((n, st), (n[::-1], [np.transpose(st[c], (2, 1, 0)) for c in (2, 1, 0, 5, 4, 3)])):
        g = Suspension(_params(m), [0, 0, 0])
        pad = 2 * (m[2] // 2 + 1)
        arr = []
        for a in s6:
            b = np.zeros((m[0], m[1], pad))
            b[:, :, :m[2]] = a
            arr.append(b.ravel())
        for _ in range(2):
            g.inject_random_stress(arr)
        fields.append([np.asarray(u).reshape(m[0], m[1], -1)[:, :, :m[2]] for u in g.get_velocity_field(1)])
    for c in range(3):
        a, b = fields[0][c], np.transpose(fields[1][2 - c], (2, 1, 0))
        assert np.any(a)
        # modes of the Nyquist planes are symmetrised along the halved direction only
        A, B = np.fft.fftn(a), np.fft.fftn(b)
        for d in range(3):
            i = [slice(None)] * 3
            i[d] = n[d] // 2
            A[tuple(i)] = B[tuple(i)] = 0
        assert rel_err(np.stack([A.real, A.imag]), np.stack([B.real, B.imag])) < 1e-11


@pytest.mark.parametrize("n, P", [((384, 16, 16), 0), ((40, 48, 48), 0), ((40, 48, 48), 1)])
def test_autotune_times_one_path_once(gpu, n, P):
    g = Suspension(_params(n, precision=1), [0, 0, 0])
    g.set_up_gaussians(np.linspace(0.0, 15.0, 30))
    for _ in range(3):
        v, us = g.autotune(reps=3)
        t = us[16 * P + 6:16 * P + 9]
        assert v[2 * P + 1] == 0 and t[0] > 0
        assert all(x in (-1.0, t[0]) for x in t[1:])
