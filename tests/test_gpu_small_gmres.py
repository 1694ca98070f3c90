"""The one-launch orthogonalisation of small systems (up to 16,384 unknowns: one, two or
four entries of the Krylov column per thread of a cluster of eight CTAs) at the sizes around
its edges, the separate kernels just beyond, and the smallest system (one body).  A rod of
six blobs has 24 unknowns.  The residual GMRES reports is checked against the residual of
the returned solution, formed with the saddle-point product: equal within 1e-11 of ||b|| (the
recurrence loses a few hundred roundings of the basis, 1e-14 each), so a wrong column, sum or
rotation shows; and a solve stopped by gmres_max_iter still returns its iterate with that
iteration's residual."""
import numpy as np
import pytest

from timstochrigidbodiessim_b200 import configs
from timstochrigidbodiessim_b200.fcm import Suspension

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 21, 170, 171, 341, 342, 682, 683])
@pytest.mark.parametrize("stop", [0, 9])
def test_residual(gpu, M, stop):
    p, ref, x, q, fe = configs.rod_suspension(M=M, grid=64 if M < 100 else 96, L=40.0 if M < 100 else 84.0, seed=M,
                                              noise=0, gmres_tol=1e-9, gmres_max_iter=stop or 100)
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
    st, soln, iters, rel = s.invert_saddle_point_system()
    true = np.linalg.norm(b - s.multiply_by_saddle_point_matrix(soln)) / np.linalg.norm(b)
    assert abs(true - rel) < 1e-11
    if stop and M > 2:
        assert st == 5 and iters == stop and rel > 1e-9
    elif not stop:
        assert st == 0 and iters < 100 and rel < 1e-9
