"""The one-launch orthogonalisation of small systems at its largest numbers of columns (up to
256 with the column to come, 45 KB of shared memory) and the separate kernels beyond, run to
the last column: a tolerance that no residual reaches, so that gmres_max_iter ends the solve.
The residual that GMRES reports is checked against that of the returned solution as in the
tests at few columns: equal within 1e-11 of ||b||.  Two contexts of different column numbers
are solved in turn and by two threads at once: neither's launches depend on the other's."""
import threading

import numpy as np
import pytest

from timstochrigidbodiessim_b200 import configs
from timstochrigidbodiessim_b200.fcm import Suspension

pytestmark = pytest.mark.gpu


def _system(M, columns):
    p, ref, x, q, fe = configs.rod_suspension(M=M, grid=64, L=40.0, seed=M, noise=0, gmres_tol=1e-290,
                                              gmres_max_iter=columns)
    s = Suspension(p, ref)
    s.set_bodies(x, q)
    s.set_external_forces(fe)
    s.produce_reference_matrices()
    s.fill_all_blob_pos()
    s.set_up_gaussians()
    s.calculate_forces()
    rng = np.random.default_rng(M)
    F = rng.standard_normal(3 * p.num_blobs)
    b = np.concatenate([rng.standard_normal(3 * p.num_blobs), -s.multiply_by_KT_at_midstep(F)])
    s.set_RHS(b)
    return s, b


def _check(s, b, columns):
    st, soln, iters, rel = s.invert_saddle_point_system()
    true = np.linalg.norm(b - s.multiply_by_saddle_point_matrix(soln)) / np.linalg.norm(b)
    assert st == 5 and iters == columns and abs(true - rel) < 1e-11


@pytest.mark.parametrize("columns", [200, 242, 243, 254, 255, 256, 300])
def test_last_column(gpu, columns):
    _check(*_system(40, columns), columns)


def test_contexts_of_different_column_numbers(gpu):
    sizes = (255, 245)
    systems = [_system(40, c) for c in sizes]
    for _ in range(2):
        for (s, b), c in zip(systems, sizes):
            _check(s, b, c)
    errors = []

    def solve(c):
        try:
            for _ in range(3):
                _check(*_system(40, c), c)
        except BaseException as e:  # noqa: BLE001 -- raised in the main thread below
            errors.append(e)

    threads = [threading.Thread(target=solve, args=(c,)) for c in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
