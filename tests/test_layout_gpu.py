"""The input layout stage of the four-kernel product: spins with and without the point-wise form, odd bonds, and inputs at any
8-byte (complex 16-byte) address.  The layout moves values only, so the offset input gives the very bits of the aligned one; both
follow the host product to 1e-13 of the norm (sums of at most 4 * 300 Gaussian terms)."""
import numpy as np
import pytest
import torch

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("S,cL,cR", [(1, 300, 260), (2, 256, 200), (2, 255, 201), (3, 200, 150), (4, 160, 160), (4, 161, 163), (4, 300, 201), (5, 140, 150)])
def test_layout(cuda, S, cL, cR, cplx):
    rng = np.random.default_rng(S + cL)
    f = lambda *s: np.asfortranarray(rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0.0))  # noqa: E731
    th, W, L, R = f(S, cL, cR), f(3, 3, S, S), f(cL, cL, 3), f(cR, cR, 3)
    ref = np.einsum("abm,sac,mnst,cdn->tbd", L, th, W, R, optimize=("greedy", 10**9))
    op = hb.MatVecMPOS([W], L, R, cplx=cplx)
    x = torch.from_numpy(np.ascontiguousarray(th.ravel(order="F"))).cuda()
    out = []
    for shift in (0, 1):
        buf = torch.zeros(x.numel() + 2, dtype=x.dtype, device="cuda")
        xs = buf[shift:shift + x.numel()]
        xs.copy_(x)
        y = torch.empty_like(x)
        op.MultAx(xs, y)
        out.append(y.cpu().numpy())
    op.close()
    assert np.array_equal(out[0], out[1])
    y = out[0].reshape(ref.shape, order="F")
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)
