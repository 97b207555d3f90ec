"""The one-launch product for small bonds at the edges of its blocks: bonds around the eight a' of a cluster and the four columns
of a CTA, odd bonds (8-byte copies), bonds left without columns in the last CTAs, spins 1 to 5, complex MPOs with and without an
imaginary part, inputs that are not finite, and the rule's borders, through the operator and the stateless call.

FP64 sums of at most 4 * 300 Gaussian terms: both sides stay far below 1e-13 of the norm."""
import numpy as np
import pytest

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu
PAIRS = ("greedy", 10**9)


def _case(S, cL, cR, DL, DR, cplx, wcplx=False, seed=0):
    rng = np.random.default_rng(seed + 31 * cL + cR)
    f = lambda c, *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if c else 0.0))  # noqa: E731
    W = f(wcplx, DL, DR, S, S) * (rng.random((DL, DR, S, S)) < 0.6)
    return f(cplx, S, cL, cR), np.asfortranarray(W.astype(np.complex128 if cplx else np.float64)), f(cplx, cL, cL, DL), f(cplx, cR, cR, DR)


def _check(S, cL, cR, DL, DR, cplx, wcplx=False):
    th, W, L, R = _case(S, cL, cR, DL, DR, cplx, wcplx)
    ref = np.einsum("abm,sac,mnst,cdn->tbd", L, th, W, R, optimize=PAIRS)
    op = hb.MatVecMPOS([W], L, R, cplx=cplx)
    y = op.MultAx_host(th)
    op.close()
    out = hb.to_device(np.zeros_like(th))
    hb.matrix_vector_product(out, hb.to_device(th), th.shape, hb.to_device(W), W.shape, hb.to_device(L), L.shape, hb.to_device(R), R.shape)
    z = hb.to_host(out, th.shape)
    for v in (y, z):
        assert np.linalg.norm(v - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("cplx,wcplx", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("cL,cR", [(1, 1), (2, 3), (7, 8), (8, 7), (9, 15), (16, 16), (17, 31), (24, 33), (33, 32), (64, 63), (5, 130)])
def test_bonds(cuda, cL, cR, cplx, wcplx):
    _check(4, cL, cR, 3, 3, cplx, wcplx)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("S,DL,DR", [(1, 1, 1), (1, 3, 2), (2, 3, 3), (2, 9, 9), (3, 2, 5), (4, 9, 9), (4, 1, 3), (5, 4, 3), (16, 3, 3)])
def test_spins_and_mpos(cuda, S, DL, DR, cplx):
    for cL, cR in [(12, 12), (13, 10), (21, 36)]:
        _check(S, cL, cR, DL, DR, cplx)


@pytest.mark.parametrize("S,cL,cR,D,cplx", [(4, 96, 96, 3, False), (4, 97, 96, 3, False), (4, 98, 98, 3, False), (4, 128, 128, 3, False), (2, 124, 93, 3, False),
                                            (2, 96, 128, 3, True), (4, 252, 5, 3, True), (4, 200, 5, 3, True), (4, 56, 56, 3, True), (4, 112, 39, 9, False)])
def test_borders_of_the_rule(cuda, S, cL, cR, D, cplx):
    _check(S, cL, cR, D, D, cplx)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_zero_weights_do_not_touch_their_inputs(cuda, cplx, value):
    S, cL, cR = 4, 11, 9
    th, _, L, R = _case(S, cL, cR, 3, 3, cplx)
    W = hb.two_site_ising_mpo(3, cplx)
    th[1, 7, 4] = value
    op = hb.MatVecMPOS([W], L, R, cplx=cplx)
    y = op.MultAx_host(th)
    op.close()
    with np.errstate(invalid="ignore"):
        T1 = np.einsum("abm,sac->mbsc", L, th)
        T2 = np.zeros((3, S, cL, cR), dtype=y.dtype)
        for m, n, s, t in zip(*np.nonzero(W)):
            T2[n, t] += W[m, n, s, t] * T1[m, :, s, :]
        ref = np.einsum("ntbc,cdn->tbd", T2, R)
    bad = ~np.isfinite(ref)
    assert bad.any() and np.array_equal(bad, ~np.isfinite(y))
    assert np.linalg.norm(y[~bad] - ref[~bad]) <= 1e-13 * np.linalg.norm(ref[~bad])
