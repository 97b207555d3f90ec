"""Device SVD of matrices of at most 17 columns at the edges of its paths: Jacobi on the matrix itself up to 64 rows, on the factor of
one panel beyond (to 16 columns, to 9 from 257 rows on, one CTA and a cluster), after two factorisations else, tall and wide, with zero columns, repeated columns, extreme scales and
a NaN.

Bars as for the other sizes (LAPACK gesdd on the host): singular values to 1e-13 sigma_max, orthonormal factors to
1e-13 max(m, n), the truncated product to 1e-12 ||A||, equal ranks."""
import numpy as np
import pytest

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu

SHAPES = [(64, 1), (65, 1), (300, 1), (64, 5), (65, 5), (64, 16), (65, 16), (64, 17), (65, 17), (256, 1), (257, 1), (256, 10), (257, 10), (256, 16), (257, 9), (288, 7), (289, 12), (673, 16), (1000, 3), (3000, 15), (5376, 9)]


def _random(m, n, cplx, graded, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0.0)
    if graded:
        U, S, V = np.linalg.svd(A, full_matrices=False)
        A = (U * np.exp(-27.0 * np.arange(len(S)) / len(S))) @ V
    return np.asfortranarray(A)


def _svd(A, **kw):
    m, n = A.shape
    U, S, VT, k, err = hb.svd(hb.to_device(A), m, n, **kw)
    return hb.to_host(U, (m, k)), S.cpu().numpy()[:k], hb.to_host(VT, (k, n)), k, err


@pytest.mark.parametrize("graded", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("m,n", SHAPES)
def test_shapes(cuda, m, n, wide, cplx, graded):
    if cplx and m > 3584:
        m = 3584
    A = _random(m, n, cplx, graded, 3 * m + n)
    if wide:
        A = np.asfortranarray(A.T)
    U, S, VT, k, err = _svd(A, rank_max=max(1, n // 2) if graded else 0, trunc_lim=1e-12)
    Ur, Sr, Vr = np.linalg.svd(A, full_matrices=False)
    assert k == (max(1, n // 2) if graded else n)
    assert np.max(np.abs(S - Sr[:k])) <= 1e-13 * Sr[0]
    assert np.linalg.norm(U.conj().T @ U - np.eye(k)) < 1e-13 * m
    assert np.linalg.norm(VT @ VT.conj().T - np.eye(k)) < 1e-13 * m
    assert np.linalg.norm(U * S @ VT - (Ur[:, :k] * Sr[:k]) @ Vr[:k]) <= 1e-12 * np.linalg.norm(A)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [(40, 12), (100, 12), (700, 16)])
def test_zero_and_repeated_columns(cuda, m, n, cplx):
    """A zero column gives an exactly zero singular value; a repeated one, or one a thousandth of another, a value at rounding level."""
    A = _random(m, n, cplx, False, n)
    A[:, [0, 5, n - 1]] = 0.0
    U, S, VT, k, err = _svd(A, trunc_lim=0.0)
    assert k == n - 3 and err == 0.0
    A[:, 5], A[:, 0] = A[:, 1], A[:, 2] / 1000
    U, S, VT, k, err = _svd(A, trunc_lim=1e-12)
    assert k == n - 3
    assert np.max(np.abs(S - np.linalg.svd(A, compute_uv=False)[:k])) <= 1e-13 * S[0]
    assert np.linalg.norm(U * S @ VT - A) <= 1e-12 * np.linalg.norm(A)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("scale", [2.0**-400, 2.0**400])
def test_scales(cuda, scale, cplx):
    A = _random(100, 10, cplx, True, 1)
    s, t = _svd(A, rank_max=5, trunc_lim=0.0)[1], _svd(A * scale, rank_max=5, trunc_lim=0.0)[1]
    assert np.max(np.abs(t / scale - s)) <= 1e-13 * s[0]


@pytest.mark.parametrize("col", [0, 3, 7])
@pytest.mark.parametrize("m", [30, 100, 700])
def test_nan_is_refused(cuda, m, col):
    A = _random(m, 8, False, False, m)
    A[m // 2, col] = np.nan
    with pytest.raises(hb.HeffError) as e:
        hb.svd(hb.to_device(A), m, 8)
    assert e.value.code == 7


def test_time_of_long_matrices(cuda):
    """One panel's factorisation (about 1.3 us a column, 60 us with its launches) brings 256 rows down to 8: the split then takes less
    than twice that of 64 rows, which fit shared memory; sweeps over all 256 rows took 2.4 times as long."""
    import torch

    us = {}
    for m in (64, 256):
        d = hb.to_device(_random(m, 8, True, True, 5))
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = []
        for _ in range(12):
            torch.cuda.synchronize()
            ev[0].record()
            hb.svd(d, m, 8, trunc_lim=0.0)
            ev[1].record()
            torch.cuda.synchronize()
            best.append(1e3 * ev[0].elapsed_time(ev[1]))
        us[m] = min(best)
    assert us[256] < 1.8 * us[64], us
