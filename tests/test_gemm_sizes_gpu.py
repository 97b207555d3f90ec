"""FP64 DMMA GEMM at the edges of its tiles and K splits, below the sizes at which a matvec reaches it: the environment updates
call it at every size (products over the batch of MPO channels, A^T B and A B^T forms, K shorter than one k-tile).

FP64 on both sides; every output is three nested sums, their K together at most 2 * 129 + 2 * 9 + 129 terms, whose errors stay
below eps K = 1e-13 of the norms."""
import numpy as np
import pytest

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu
PAIRS = ("greedy", 10**9)


@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("D", [1, 3, 9])
@pytest.mark.parametrize("cL,cR", [(1, 1), (7, 5), (31, 33), (32, 32), (33, 31), (48, 3), (3, 48), (63, 65), (64, 64), (65, 63), (127, 129), (128, 128), (129, 127)])
def test_env_at_tile_edges(cuda, side, cL, cR, D, cplx):
    rng = np.random.default_rng(cL * 131 + cR)
    f = lambda *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0.0))  # noqa: E731
    M, W = f(2, cL, cR), f(D, D, 2, 2)
    E = f(cL, cL, D) if side == "L" else f(cR, cR, D)
    shape = (cR, cR, D) if side == "L" else (cL, cL, D)
    dE, dM, dW = hb.to_device(E), hb.to_device(M), hb.to_device(W)
    outs = []
    for _ in range(2):
        out = hb.to_device(np.full(shape, np.nan, dtype=E.dtype, order="F"))
        hb.env_update(side, out, dE, E.shape, dM, M.shape, dW, W.shape)
        outs.append(hb.to_host(out, shape))
    expr = "abm,sac,tbd,mnst->cdn" if side == "L" else "cdn,sac,tbd,mnst->abm"
    ref = np.einsum(expr, E, M, M.conj(), W, optimize=PAIRS)
    assert np.linalg.norm(outs[0] - ref) <= 1e-13 * np.linalg.norm(ref)
    assert np.array_equal(outs[0], outs[1])  # a fixed order of every sum
