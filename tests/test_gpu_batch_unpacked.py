"""Batches and single contexts on grids that the packed half spectrum does not take: a side of
88 points along y (the fused x-transform between cuFFT's (y, z) plans of the whole group) and
along x (cuFFT's 3D plans of the group and k_b_project), a group of each beside a packed one
in the same batch.  Members follow the same suspensions stepped alone (1e-9 in FP64, 1e-8 mixed:
the tolerances of the other batch tests).  And single contexts whose x length has the fused
x-transform but whose y or z length is not a packed one: the solve variants against the
oracle (1e-10 in FP64, 1e-6 in FP32, as the other variants)."""
import numpy as np
import pytest

from tests.conftest import rel_err
from tests.oracle_lib import Oracle
from timstochrigidbodiessim_b200 import configs
from timstochrigidbodiessim_b200.fcm import Batch, Suspension
from timstochrigidbodiessim_b200.params import FcmParams, rod_reference_positions

pytestmark = pytest.mark.gpu


def _rods(n, M, seed, precision, algorithm):
    """M rods of three blobs on a lattice of a box of n points, far enough apart not to touch."""
    ref = np.array(rod_reference_positions(3, 2.2))
    p = FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=12, dx=0.5, num_bodies=M, blobs_per_body=3, ncells=3,
                           potential=3, gmres_tol=1e-8 if precision else 1e-10, gmres_max_iter=100,
                           precision=precision, algorithm=algorithm, dt=0.01)
    rng = np.random.default_rng(seed)
    box = 0.5 * np.array(n)
    m = np.floor(box / 8.0).astype(int)
    site = rng.permutation(int(m.prod()))[:M]
    ijk = np.stack([site // (m[1] * m[2]), (site // m[2]) % m[1], site % m[2]], axis=1)
    x = ((ijk + 0.5) * box / m + rng.uniform(-0.3, 0.3, (M, 3))).ravel()
    q = configs.random_unit_quaternions(rng, M).ravel()
    fe = np.zeros(6 * M)
    fe[2::6] = -1.0
    return p, ref, x, q, fe


@pytest.mark.parametrize("precision, algorithm", [(0, 2), (1, 2), (1, 1)])
@pytest.mark.parametrize("grids", [[(96, 88, 64)] * 3, [(88, 88, 88)] * 2, [(88, 64, 64), (64, 64, 88)],
                                   [(96, 88, 64), (64, 64, 64), (88, 88, 88), (64, 64, 64), (88, 88, 88), (96, 88, 64)]])
def test_members_follow_single_steps(gpu, grids, precision, algorithm):
    insts = [_rods(n, 12 + 5 * i, i, precision, algorithm) for i, n in enumerate(grids)]
    solo = []
    for p, ref, x, q, fe in insts:
        s = Suspension(p, ref)
        solo.append(s)
    b = Batch([(p, ref) for p, ref, *_ in insts])
    for group in (solo, b.members):
        for s, (p, ref, x, q, fe) in zip(group, insts):
            s.set_bodies(x, q)
            s.set_external_forces(fe)
            s.produce_reference_matrices()
    seeds = list(range(5, 5 + len(insts)))
    for k in range(3):
        infos = b.step(seeds, k)
        for i, s in enumerate(solo):
            st, inf = s.step(seeds[i], k)
            assert st == 0 and infos[i].status == 0
            assert abs(inf.gmres_iters - infos[i].gmres_iters) <= 1, (k, i)
    tol = 1e-8 if precision == 1 else 1e-9
    for i, (s, m) in enumerate(zip(solo, b.members)):
        for a, c in zip(s.get_bodies(), m.get_bodies()):
            assert np.max(np.abs(a - c)) <= tol, i
        assert np.max(np.abs(s.get_bodies()[0] - insts[i][2])) > 1e-3
    b.close()


@pytest.mark.parametrize("n", [(12, 16, 10), (64, 22, 16), (256, 22, 16), (256, 16, 44), (384, 22, 16), (512, 16, 26)])
def test_fused_x_transform_of_single_contexts(gpu, n):
    nb = 24
    p = FcmParams.defaults(nx=n[0], ny=n[1], nz=n[2], ngauss=8, dx=1.0, num_bodies=nb, blobs_per_body=1, ncells=3,
                           precision=1)
    rng = np.random.default_rng(sum(n))
    Y = (rng.uniform(0, 1, (nb, 3)) * np.array(n)).ravel()
    F = rng.standard_normal(3 * nb)
    g, o = Suspension(p, [0, 0, 0]), Oracle(p.copy(precision=0), [0, 0, 0])
    for s in (g, o):
        s.set_up_gaussians(Y)
    ref = o.apply_mobility(F)
    v = g.get_variants()
    assert v[1] == (0 if n[0] > 256 else 1) and v[3] == 1
    for prec in (0, 1):
        out = []
        for sv in (0, 1):
            v[2 * prec + 1] = sv
            g.set_variants(v)
            g.spread(F, prec)
            g.stokes_solve(prec)
            out.append(g.interp(prec).copy())
            assert rel_err(out[-1], ref) < (1e-6 if prec else 1e-10), (prec, sv)
        assert not np.array_equal(out[0], out[1])  # two paths, not one
