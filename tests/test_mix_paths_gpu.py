"""MPO mix at sizes that the one-launch product does not take (shown by the launch counter): point counts around its tiles, spins
with unpaired outputs, MPOs of more fragments than the two-site Ising square, inputs that are not finite in tiles of 32, 64 and
128 points with one and two tiles in flight, and environment MPOs whose inputs fit no tile.

The host products are FP64 einsums; the sums have at most 3 * 400 + 80 Gaussian terms each, errors far below 1e-13 of the norm."""
import numpy as np
import pytest

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu
PAIRS = ("greedy", 10**9)


def _case(S, cL, cR, DL, DR, cplx, wcplx=False, density=0.3, seed=0):
    rng = np.random.default_rng(seed + 17 * cL + cR)
    f = lambda c, *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if c else 0.0))  # noqa: E731
    W = f(wcplx, DL, DR, S, S) * (rng.random((DL, DR, S, S)) < density)
    W[-1, -1, -1, -1] = 1.0
    return f(cplx, S, cL, cR), np.asfortranarray(W.astype(np.complex128 if cplx else np.float64)), f(cplx, cL, cL, DL), f(cplx, cR, cR, DR)


def _matvec(th, W, L, R):
    op = hb.MatVecMPOS([W], L, R, cplx=np.iscomplexobj(th))
    n0 = hb.lib().heff_matvec_launches()
    y = op.MultAx_host(th)
    assert hb.lib().heff_matvec_launches() - n0 >= 4  # layout, GEMM, mix, GEMM: not the one-launch product
    op.close()
    return y


@pytest.mark.parametrize("cplx,wcplx", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("S,DL,DR", [(1, 1, 1), (1, 5, 3), (2, 3, 3), (3, 4, 2), (4, 1, 9), (4, 3, 1), (5, 7, 6), (2, 40, 8), (16, 3, 3), (8, 6, 6), (4, 12, 12), (2, 25, 25)])
def test_shapes(cuda, S, DL, DR, cplx, wcplx):
    if cplx and S * DL >= 80:
        pytest.skip("complex MPOs above 200 KB with 128 points of input are refused")
    for cL, cR in [(331, 259), (260, 258)]:
        th, W, L, R = _case(S, cL, cR, DL, DR, cplx, wcplx)
        ref = np.einsum("abm,sac,mnst,cdn->tbd", L, th, W, R, optimize=PAIRS)
        assert np.linalg.norm(_matvec(th, W, L, R) - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("cL", [280, 290, 380])  # tiles of 32, 64 and 128 points
@pytest.mark.parametrize("cplx,wcplx", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("D", [3, 9])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_zero_weights_do_not_touch_their_inputs(cuda, cL, D, cplx, wcplx, value):
    """A non-finite theta entry of spin 1 reaches the outputs that W's nonzero entries lead to, and no other."""
    S, cR = 4, 300
    th, W, L, R = _case(S, cL, cR, D, D, cplx, wcplx, density=0.1, seed=D)
    W[:, :, 1, 0] = W[:, :, 1, 3] = 0.0
    W[D - 1, 0, 1, 2] = 2.0
    th[1, 7, 4] = value
    y = _matvec(th, W, L, R)
    hit = [bool(np.any(W[:, :, 1, t] != 0)) for t in range(S)]
    for t in range(S):
        assert np.all(np.isfinite(y[t])) if not hit[t] else not np.any(np.isfinite(y[t]))
    th[1, 7, 4] = 0.0
    ref = np.einsum("abm,sac,mnst,cdn->tbd", L, th, W, R, optimize=PAIRS)
    for t in range(S):
        if not hit[t]:
            assert np.linalg.norm(y[t] - ref[t]) <= 1e-13 * np.linalg.norm(ref[t])


def _env(side, E, M, W):
    shape = (M.shape[2], M.shape[2], W.shape[1]) if side == "L" else (M.shape[1], M.shape[1], W.shape[0])
    out = hb.to_device(np.zeros(shape, dtype=E.dtype, order="F"))
    hb.env_update(side, out, hb.to_device(E), E.shape, hb.to_device(M), M.shape, hb.to_device(W), W.shape)
    expr = "abm,sac,tbd,mnst->cdn" if side == "L" else "cdn,sac,tbd,mnst->abm"
    return hb.to_host(out, shape), lambda e: np.einsum(expr, e, M, M.conj(), W, optimize=PAIRS)


@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("cplx", [False, True])
def test_env_zero_weights_do_not_touch_their_inputs(cuda, side, cplx):
    """An environment entry of channel 1 that is not finite reaches the output channels that W couples to it only."""
    rng = np.random.default_rng(3)
    f = lambda *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0.0))  # noqa: E731
    M, W, E = f(2, 37, 37), f(3, 3, 2, 2), f(37, 37, 3)
    free = (W[1], W[:, 1])[side == "R"]  # the entries that channel 1 meets, output channel first
    free[0] = free[2] = 0.0
    E[5, 7, 1] = np.nan
    y, ref = _env(side, E, M, W)
    E[5, 7, 1] = 0.0
    r = ref(E)
    assert not np.any(np.isfinite(y[:, :, 1]))
    for n in (0, 2):
        assert np.linalg.norm(y[:, :, n] - r[:, :, n]) <= 1e-13 * np.linalg.norm(r[:, :, n])


@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("d,Din,Dout", [(2, 1024, 1), (1, 2048, 2), (2, 340, 3), (2, 1, 1024), (2, 32, 32), (4, 16, 16)])
def test_env_long_mpo_bonds(cuda, side, d, Din, Dout, cplx):
    rng = np.random.default_rng(Din)
    f = lambda *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0.0))  # noqa: E731
    DL, DR = (Din, Dout) if side == "L" else (Dout, Din)
    M, W = f(d, 9, 11), f(DL, DR, d, d) * (rng.random((DL, DR, d, d)) < 0.3)
    c = 9 if side == "L" else 11
    E = f(c, c, Din)
    y, ref = _env(side, E, M, W)
    r = ref(E)
    assert np.linalg.norm(y - r) <= 1e-13 * np.linalg.norm(r)


def test_mix_time_grows_with_its_products(cuda):
    """The mix of an MPO with 128 fragments (S = 4, D = 16) does 2.8 times the products of one with 45 (D = 9) and moves 1.8 times the
    bytes; walking its entries from global memory took tens of times as long."""
    us = {}
    for D in (9, 16):
        th, W, L, R = _case(4, 128, 128, D, D, False, density=0.2)
        op = hb.MatVecMPOS([W], L, R)
        x = hb.to_device(th)
        y = hb.to_device(np.zeros_like(th))
        for _ in range(3):
            op.MultAx(x, y)
        op.set_profiling(True)
        for _ in range(20):
            op.MultAx(x, y)
        ms, n = op.stage_times()
        us[D] = 1e3 * ms[2] / n
        op.close()
    assert us[16] < 6.0 * us[9], us
