"""The Jacobi rotations of the device SVD are right to double precision: one rotation diagonalises a 2 x 2 Gram to a few eps (its
singular values are within a factor of ten here, so below the test's 1e-14), and the sweep after it finds nothing to rotate.  An
angle from a shorter format leaves its residue to a third sweep."""
import numpy as np
import pytest

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
def test_two_columns_take_one_rotation(cuda, seed):
    h = np.random.default_rng(seed).uniform(0.5, 1.5, 2)
    r = hb.fdmrg(h, chi_max=2, sweeps=1)  # two sites: every split is of a 2 x 2 matrix
    # Schmidt values of the ground state of -s1 s2 - h.sx on two sites
    sx, sz, one = np.array([[0, 1], [1, 0]]), np.diag([1, -1]), np.eye(2)
    w, v = np.linalg.eigh(-np.kron(sz, sz) - h[0] * np.kron(sx, one) - h[1] * np.kron(one, sx))
    s = np.linalg.svd(v[:, 0].reshape(2, 2), compute_uv=False)
    assert abs(r["energy"] - w[0]) < 1e-12 and s[1] > 0.1 * s[0]
    assert r["svd_sweeps_max"] <= 2
