"""Device SVD at the edges of its paths: plain and QR-preconditioned Jacobi (16 / 17 columns), one-CTA Jacobi of 32 and 64
columns and the pair rounds beyond, matrices longer than a resident tile or a panel of one CTA, longer than a preconditioned
panel can be, wide ones, zero columns, and scales at which the squares of the entries leave double precision's range.

Bars as for the other sizes (LAPACK gesdd on the host): singular values to 1e-13 sigma_max, orthonormal factors to
1e-13 max(m, n), the truncated product to 1e-12 ||A||, equal ranks."""
import numpy as np
import pytest
import torch

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (2, 1), (1, 3), (16, 16), (17, 17), (16, 257), (257, 16), (256, 16), (31, 33), (32, 32), (33, 33), (65, 32), (64, 64), (65, 64),
          (64, 66), (65, 65), (70, 172), (300, 64), (97, 90), (129, 96), (700, 40), (1500, 100), (45, 1400)]


def _check(A, rank_max=0, lim=1e-12):
    m, n = A.shape
    U, S, VT, k, err = hb.svd(hb.to_device(A), m, n, rank_max=rank_max, trunc_lim=lim)
    Ur, Sr, Vr = np.linalg.svd(A, full_matrices=False)
    tail = np.sqrt(np.cumsum(Sr[::-1] ** 2)[::-1])
    kr = min(int(np.sum(tail >= lim)), rank_max or len(Sr))
    assert k == kr
    U, VT, S = hb.to_host(U, (m, k)), hb.to_host(VT, (k, n)), S.cpu().numpy()
    assert np.max(np.abs(S - Sr[:k])) <= 1e-13 * Sr[0]
    assert np.linalg.norm(U.conj().T @ U - np.eye(k)) < 1e-13 * max(m, n)
    assert np.linalg.norm(VT @ VT.conj().T - np.eye(k)) < 1e-13 * max(m, n)
    assert np.linalg.norm(U * S @ VT - (Ur[:, :k] * Sr[:k]) @ Vr[:k]) <= 1e-12 * np.linalg.norm(A)
    assert abs(err - (tail[k] if k < len(Sr) else 0.0)) <= 1e-13 * Sr[0]


def _random(m, n, cplx, graded, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0.0)
    if graded:
        U, S, V = np.linalg.svd(A, full_matrices=False)
        A = (U * np.exp(-27.0 * np.arange(len(S)) / len(S))) @ V
    return np.asfortranarray(A)


@pytest.mark.parametrize("graded", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", SHAPES)
def test_path_edges(cuda, m, n, cplx, graded):
    A = _random(m, n, cplx, graded, 3 * m + n)
    _check(A, rank_max=max(1, min(m, n) // 2) if graded else 0, lim=1e-12)


@pytest.mark.parametrize("m,n,cplx", [(5376, 17, False), (5377, 17, False), (3585, 20, True)])
def test_longest_panels(cuda, m, n, cplx):
    _check(_random(m, n, cplx, True, m), rank_max=n // 2)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [12, 40, 80])
def test_zero_columns_and_no_truncation(cuda, n, cplx):
    """A zero column gives an exactly zero singular value, which the rank rule does not count even without a limit."""
    A = _random(n + 7, n, cplx, False, n)
    A[:, [0, 5, n - 1]] = 0.0
    U, S, VT, k, err = hb.svd(hb.to_device(A), n + 7, n, trunc_lim=0.0)
    assert k == n - 3 and err == 0.0
    assert np.max(np.abs(S.cpu().numpy() - np.linalg.svd(A, compute_uv=False)[: n - 3])) < 1e-13 * n


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [10, 40, 80])
@pytest.mark.parametrize("scale", [2.0**-400, 2.0**400])
def test_scales(cuda, n, scale, cplx):
    """A power of two changes nothing but the exponent: the same factors, the singular values scaled."""
    A = _random(n, n, cplx, True, n)
    U, S, VT, k, _ = hb.svd(hb.to_device(A), n, n, rank_max=n // 2, trunc_lim=0.0)
    Us, Ss, VTs, ks, _ = hb.svd(hb.to_device(A * scale), n, n, rank_max=n // 2, trunc_lim=0.0)
    assert ks == k
    s = S.cpu().numpy()
    assert np.max(np.abs(Ss.cpu().numpy() / scale - s)) <= 1e-13 * s[0]
    prod = hb.to_host(U, (n, k)) * s @ hb.to_host(VT, (k, n))
    prods = hb.to_host(Us, (n, k)) * (Ss.cpu().numpy() / scale) @ hb.to_host(VTs, (k, n))
    assert np.linalg.norm(prod - prods) <= 1e-12 * s[0]


def test_nan_is_refused(cuda):
    for n in (8, 40, 80):
        A = _random(n, n, False, False, n)
        A[n // 2, 1] = np.nan
        with pytest.raises(hb.HeffError) as e:
            hb.svd(hb.to_device(A), n, n)
        assert e.value.code == 7
    torch.cuda.synchronize()
