"""The Krylov expansion step in one launch, through the eigensolver: vector lengths around the rows that eight and sixteen CTAs hold
and around the border to the three-launch form, bases across the 8, 16 and 24 column forms.

The solver declares convergence on an explicit residual of tol * ||H||, so ||H x - e x|| <= 1e-11 ||H|| up to the rounding of an
FP64 product (1e-13 ||H||), and two converged runs of the same state differ in energy by at most the sum of their residuals."""
import numpy as np
import pytest
import torch

import dmrg_b200 as hb
from oracle import physics as ph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cL,cR,cplx", [(5, 4, False), (32, 32, False), (32, 33, False), (64, 63, False), (128, 64, False), (128, 65, False),
                                        (5, 4, True), (32, 16, True), (32, 17, True), (64, 64, True), (64, 65, True)])
def test_one_launch_orthonormalisation(cuda, cL, cR, cplx):
    th, W, L, R = ph.heff_inputs(cL, D=3, cplx=cplx, seed=3, chiR=cR)
    op = hb.MatVecMPOS([W], L, R, cplx=cplx)
    x0 = torch.from_numpy(np.ascontiguousarray(th.ravel(order="F"))).cuda()
    e = []
    for max_basis in (24, 9, 40):  # 40: columns beyond 24 take the general kernels
        x = torch.empty_like(x0)
        val, res = op.eigs(x0=x0, x_out=x, tol=1e-11, max_basis=max_basis, min_basis=4)
        assert res["converged"] == 1
        y = torch.empty_like(x)
        op.MultAx(x, y)
        scale = float(torch.linalg.vector_norm(y)) + abs(op.eigs(x0=x0, ritz="LA", tol=1e-3)[0])  # at least ||H||
        assert abs(float(torch.linalg.vector_norm(x)) - 1.0) < 1e-12
        assert float(torch.linalg.vector_norm(y - val * x)) <= 1.1e-11 * scale
        e.append((val, scale))
    for val, scale in e[1:]:
        assert abs(val - e[0][0]) <= 2.2e-11 * scale
    op.close()
