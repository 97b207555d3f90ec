"""MPO mix (the middle stage of the matvec and of the environment updates) at the edges of its paths: point counts around the
tiles of 32, 64 and 128, odd extents (8-byte copies), spins with unpaired outputs, complex MPOs with and without an imaginary
part, bonds too long for the dense product, and inputs that are not finite.

The host products are FP64 einsums; K S <= 640 terms of Gaussian data keep both errors far below 1e-13 of the norm."""
import numpy as np
import pytest

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu
PAIRS = ("greedy", 10**9)  # pairwise contractions, whatever the size of their intermediates


def _case(S, cL, cR, DL, DR, cplx, wcplx=None, density=0.4, seed=0):
    rng = np.random.default_rng(seed + 17 * cL + cR)
    f = lambda c, *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if c else 0.0))  # noqa: E731
    W = f(cplx if wcplx is None else wcplx, DL, DR, S, S) * (rng.random((DL, DR, S, S)) < density)
    dt = np.complex128 if cplx else np.float64
    return f(cplx, S, cL, cR), np.asfortranarray(W.astype(dt)), f(cplx, cL, cL, DL), f(cplx, cR, cR, DR)


def _matvec(th, W, L, R):
    op = hb.MatVecMPOS([W], L, R, cplx=np.iscomplexobj(th))
    y = op.MultAx_host(th)
    op.close()
    return y


def _close(a, b):  # a random MPO of one element may be zero: the product is then zero too
    return np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)


@pytest.mark.parametrize("cplx,wcplx", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("S,DL,DR", [(1, 1, 1), (1, 5, 3), (2, 3, 3), (3, 4, 2), (4, 3, 3), (4, 9, 9), (4, 1, 9), (4, 3, 1), (5, 7, 6), (2, 40, 8), (4, 30, 5)])
def test_mix_shapes(cuda, S, DL, DR, cplx, wcplx):
    for cL, cR in [(1, 3), (33, 31), (130, 9)]:
        th, W, L, R = _case(S, cL, cR, DL, DR, cplx, wcplx)
        if cplx and S * DL >= 80:  # complex MPOs above 200 KB with 128 points of input are refused
            with pytest.raises(hb.HeffError, match="HEFF_BAD_SHAPE"):
                _matvec(th, W, L, R)
            continue
        ref = np.einsum("abm,sac,mnst,cdn->tbd", L, th, W, R, optimize=PAIRS)
        assert _close(_matvec(th, W, L, R), ref)


@pytest.mark.parametrize("cL,cR", [(31, 300), (32, 300), (64, 200), (65, 150), (127, 300), (128, 300), (129, 299), (517, 20)])
def test_mix_tiles(cuda, cL, cR):
    for cplx in (False, True):
        th, W, L, R = _case(4, cL, cR, 3, 3, cplx, False)
        ref = np.einsum("abm,sac,mnst,cdn->tbd", L, th, W, R, optimize=PAIRS)
        assert _close(_matvec(th, W, L, R), ref)


@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("d,cL,cR,DL,DR", [(2, 33, 45, 3, 3), (2, 130, 64, 9, 9), (3, 21, 20, 4, 5), (1, 40, 33, 2, 2), (2, 20, 21, 100, 10)])
def test_env_mix_shapes(cuda, side, d, cL, cR, DL, DR, cplx):
    rng = np.random.default_rng(d + cL)
    f = lambda *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0.0))  # noqa: E731
    M, W = f(d, cL, cR), f(DL, DR, d, d) * (rng.random((DL, DR, d, d)) < 0.5)
    E = f(cL, cL, DL) if side == "L" else f(cR, cR, DR)
    shape = (cR, cR, DR) if side == "L" else (cL, cL, DL)
    out = hb.to_device(np.zeros(shape, dtype=E.dtype, order="F"))
    hb.env_update(side, out, hb.to_device(E), E.shape, hb.to_device(M), M.shape, hb.to_device(W), W.shape)
    if side == "L":
        ref = np.einsum("abm,sac,tbd,mnst->cdn", E, M, M.conj(), W, optimize=PAIRS)
    else:
        ref = np.einsum("cdn,sac,tbd,mnst->abm", E, M, M.conj(), W, optimize=PAIRS)
    assert _close(hb.to_host(out, shape), ref)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_zero_weights_do_not_touch_their_inputs(cuda, cplx, value):
    """A non-finite theta entry reaches exactly the outputs that a product over the nonzero MPO entries gives."""
    S, cL, cR = 4, 20, 9
    th, _, L, R = _case(S, cL, cR, 3, 3, cplx)
    W = hb.two_site_ising_mpo(3, cplx)
    th[1, 7, 4] = value
    y = _matvec(th, W, L, R)
    with np.errstate(invalid="ignore"):
        T1 = np.einsum("abm,sac->mbsc", L, th)
        T2 = np.zeros((3, S, cL, cR), dtype=y.dtype)
        for m, n, s, t in zip(*np.nonzero(W)):
            T2[n, t] += W[m, n, s, t] * T1[m, :, s, :]
        ref = np.einsum("ntbc,cdn->tbd", T2, R)
    bad = ~np.isfinite(ref)
    assert bad.any() and not bad.all()
    assert np.array_equal(bad, ~np.isfinite(y))
    assert np.linalg.norm((y[~bad] - ref[~bad])) < 1e-13 * np.linalg.norm(ref[~bad])
