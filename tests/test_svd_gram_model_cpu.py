"""Host model of the one-CTA device SVD (oracle.ref_numpy.jacobi_gram_model: the factorisations, Gram per sweep, rotations from half
of the convergence test's thresholds, the kernels' rotation formula) against LAPACK, on the reference's own SVD inputs and on
Gaussian and graded matrices: singular values within 1e-14 sigma_max sqrt(n), the right factor orthonormal to 1e-13 n, the product to
1e-13 ||A|| (a few eps per sweep of at most n rotations a column), and few sweeps.  The left factor is orthonormal as far as the
criterion asks: a pair passes with |y_i^H y_j| <= max(tol s_i s_j, floor), floor = n eps^2 s_0^2.  The rotation itself: unitary to a few eps for
every angle, and what it leaves of the off-diagonal is rounding, not the residue of a shorter format."""
import glob
import os

import numpy as np
import pytest

from dmrg_b200 import replay
from oracle import ref_numpy as rn

FIX = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "reference_h5")
EPS = 2.220446049250313e-16


def _reference():
    for p in sorted(glob.glob(os.path.join(FIX, "svd*.h5"))):
        for d in replay.svd_dumps(p):
            if min(d["A"].shape) <= 64:
                yield pytest.param(d["A"], id=f"{os.path.basename(p)}:{d['name']}")


def _made():
    for cplx in (False, True):
        for m, n in [(1, 1), (3, 2), (12, 12), (100, 7), (70, 1), (300, 1), (300, 16), (17, 17), (40, 33), (33, 40), (64, 64)]:
            rng = np.random.default_rng(m + n)
            A = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0.0)
            yield pytest.param(A, id=f"gauss-{m}x{n}-{'c' if cplx else 'r'}")
            U, S, V = np.linalg.svd(A, full_matrices=False)
            yield pytest.param((U * np.exp(-27.0 * np.arange(len(S)) / len(S))) @ V, id=f"graded-{m}x{n}-{'c' if cplx else 'r'}")


@pytest.mark.parametrize("A", [*_reference(), *_made()])
def test_model(A):
    U, s, V, sweeps = rn.jacobi_gram_model(A)
    n = min(A.shape)
    ref = np.linalg.svd(A, compute_uv=False)
    assert sweeps <= 12
    assert np.max(np.abs(s - ref)) <= 1e-14 * np.sqrt(n) * max(ref[0], 1e-300)
    wide = A.shape[0] < A.shape[1]
    left, right = (V, U) if wide else (U, V)
    assert np.linalg.norm(right.conj().T @ right - np.eye(n)) <= 1e-13 * n
    k = int(np.sum(s > 0))
    bound = np.maximum(1e-14 * np.sqrt(max(A.shape)), max(A.shape) * EPS**2 * s[0] ** 2 / np.outer(s[:k], s[:k])) + 1e-14 * n
    assert np.all(np.abs(left[:, :k].conj().T @ left[:, :k] - np.eye(k)) <= bound)
    assert np.linalg.norm((U * s) @ V.conj().T - A) <= 1e-13 * np.linalg.norm(A)


@pytest.mark.parametrize("cplx", [False, True])
def test_rotation(cplx):
    rng = np.random.default_rng(1)
    for _ in range(2000):
        X = rng.standard_normal((6, 2)) + (1j * rng.standard_normal((6, 2)) if cplx else 0.0)
        X[:, 1] = X[:, 1] * 10.0 ** rng.uniform(-3, 0) + X[:, 0] * 10.0 ** rng.uniform(-6, 1)
        G = X.conj().T @ X
        p, se = rn.jacobi_rotation(G[0, 0].real, G[1, 1].real, G[0, 1], 1e-14, 0.0)
        J = np.array([[1.0 - p, se], [-np.conj(se), 1.0 - p]])
        assert np.linalg.norm(J.conj().T @ J - np.eye(2)) <= 8 * EPS
        assert abs((J.conj().T @ G @ J)[0, 1]) <= 16 * EPS * np.linalg.norm(G)
