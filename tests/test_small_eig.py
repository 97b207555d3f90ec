"""Host Rayleigh-Ritz of the Krylov loop: eigenvalues and last components against numpy, for dense, arrow-and-tridiagonal (thick
restart), diagonal and graded matrices, real and complex, at ordinary and extreme scales.

Backward stable reductions of order k <= 40: eigenvalues within 40 * 8 * 2.2e-16 < 1e-13 of the norm; the last components of
well-separated pairs (gaps of the matrices below are at least 1e-3 of the norm) within 1e-10."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dmrg_b200", "csrc")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("small_eig")
    src = d / "shim.cpp"
    src.write_text("""
#include "small_eig.hpp"
template<class T> static int run(int n, const T *a, double *d, double *z) {
    std::vector<T> A(a, a + (size_t)n * n); std::vector<double> D, Z;
    const int rc = heff::last_row_eig(n, A, D, Z);
    for(int i = 0; i < n && !rc; i++) d[i] = D[i], z[i] = Z[i];
    return rc;
}
extern "C" int eig_d(int n, const double *a, double *d, double *z) { return run(n, a, d, z); }
extern "C" int eig_z(int n, const std::complex<double> *a, double *d, double *z) { return run(n, a, d, z); }
""")
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


def _matrix(kind, n, cplx, rng):
    f = lambda *s: rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0.0)  # noqa: E731
    lam = np.linspace(-1.0, 1.0, n) if n > 1 else np.array([0.7])  # gaps of 2 / (n - 1)
    if kind == "graded":
        lam = np.sign(lam + 1e-9) * 10.0 ** (-2.0 * np.arange(n) / n)
    Q = np.linalg.qr(f(n, n))[0]
    A = (Q * lam) @ Q.conj().T
    if kind == "diagonal":
        A = np.diag(lam).astype(A.dtype)
    if kind == "arrow":  # Ritz values, couplings to the vector after them, then a tridiagonal part
        m = n // 2
        A = np.diag(lam).astype(A.dtype)
        for i in range(n - 1):
            j = m if i < m else i + 1
            if i != j:
                A[i, j] = 0.3 * f(1)[0] / n
                A[j, i] = np.conj(A[i, j])
        A += 1e-17 * f(n, n)
    return 0.5 * (A + A.conj().T)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["dense", "arrow", "diagonal", "graded"])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 24, 40])
def test_last_row(host, n, kind, cplx):
    A = _matrix(kind, n, cplx, np.random.default_rng(n))
    w, V = np.linalg.eigh(A)
    for scale in (1.0, 1e200, 1e-200):
        B = np.asfortranarray(A * scale)
        d, z = np.empty(n), np.empty(n)
        P = ctypes.c_void_p
        assert (host.eig_z if cplx else host.eig_d)(n, P(B.ctypes.data), P(d.ctypes.data), P(z.ctypes.data)) == 0
        o = np.argsort(d)
        norm = np.abs(w).max()
        assert np.abs(d[o] / scale - w).max() <= 1e-13 * norm
        gap = np.min(np.diff(w)) if n > 1 else norm
        if gap > 1e-3 * norm:
            assert np.abs(z[o] - np.abs(V[-1])).max() <= 1e-10


def test_not_finite(host):
    B = np.full((3, 3), np.nan)
    d = np.empty(3)
    assert host.eig_d(3, ctypes.c_void_p(B.ctypes.data), ctypes.c_void_p(d.ctypes.data), ctypes.c_void_p(d.ctypes.data)) != 0
