"""The dense eigensolver's matrix is shifted, its singular values lie within a factor of about 200 and need no preconditioning: a
decomposition takes less time than the preconditioned SVD of a Gaussian matrix of its size, although it also bounds the spectrum,
shifts and sorts (three launches)."""
import numpy as np
import pytest
import torch

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu


def _us(f):
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = []
    for _ in range(15):
        torch.cuda.synchronize()
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        best.append(1e3 * a.elapsed_time(b))
    return min(best)


@pytest.mark.parametrize("n", [24, 32])
def test_dense_eig_takes_less_than_an_svd(cuda, n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    H, G = hb.to_device(np.asfortranarray(G + G.conj().T)), hb.to_device(np.asfortranarray(G))
    e, s = _us(lambda: hb.dense_eig(H, n)), _us(lambda: hb.svd(G, n, n))
    assert e < 0.9 * s, (e, s)
