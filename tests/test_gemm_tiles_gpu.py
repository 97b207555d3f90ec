"""FP64 DMMA GEMM through the matvec: every tile shape and K split that its plan can pick, at the edges of the tiles.

The plan goes by size, so the sizes here sit one below, at and one above the tile edges (32, 64, 128) and k-tiles (32),
with odd leading dimensions (8-byte copies), a long K on few tiles (cluster and tail split), and K shorter than one
k-tile.  The host product is FP64 too; both errors are within a few eps sqrt(K) of the norms, K <= 2259 here, so
2e-14 covers them with an order of magnitude to spare."""
import numpy as np
import pytest

import dmrg_b200 as hb
from oracle import physics as ph
from oracle import ref_numpy as rn

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (7, 5), (31, 33), (32, 32), (33, 31), (63, 65), (64, 64), (65, 63), (97, 48), (127, 129), (128, 128), (129, 127), (200, 331),
         (48, 400), (367, 251)]


def _relerr(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("D,S", [(3, 4), (9, 4), (3, 2)])
@pytest.mark.parametrize("chiL,chiR", SIZES)
def test_matvec_at_tile_edges(cuda, chiL, chiR, D, S, cplx):
    th, W, L, R = ph.heff_inputs(chiL, D=D, cplx=cplx, seed=chiL * 7 + chiR, chiR=chiR, spin=S)
    op = hb.MatVecMPOS([W], L, R, cplx=cplx)
    y = op.MultAx_host(th)
    assert _relerr(y, rn.matvec_blas(th, W, L, R)) < 2e-14
    assert np.array_equal(y, op.MultAx_host(th))  # a fixed order of every sum
    op.close()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("mode", [0, 2, 3])
def test_split_modes_agree(cuda, mode, cplx):
    """No K split at all, and forced tail splits of the large tiles, against the automatic plan."""
    th, W, L, R = ph.heff_inputs(130, D=9, cplx=cplx, seed=5, chiR=70)
    op = hb.MatVecMPOS([W], L, R, cplx=cplx)
    y = op.MultAx_host(th)
    prev = hb.lib().heff_gemm_set_tail_split(mode)
    try:
        z = op.MultAx_host(th)
    finally:
        hb.lib().heff_gemm_set_tail_split(prev)
    assert _relerr(z, y) < 2e-14
    op.close()
