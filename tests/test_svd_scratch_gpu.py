"""Device memory of an SVD's scratch: the matrix and what its path needs, nothing kept for other shapes (a stream's workspace takes a
quarter more than asked).  A matrix too long to be factored needs itself and the square V; a tall factored one itself and three
squares, no room for the adjoint that a wide one has."""
import ctypes

import numpy as np
import pytest
import torch

import dmrg_b200 as hb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,nbytes", [(200000, 32, 8 * 200000 * 32), (5000, 1000, 8 * (5000 * 1024 + 3 * 1024**2)), (1000, 5000, 8 * (2 * 5000 * 1024 + 3 * 1024**2))])
def test_scratch(cuda, m, n, nbytes):
    rng = np.random.default_rng(1)
    k = 4
    A = hb.to_device(np.asfortranarray(rng.standard_normal((m, k)) @ rng.standard_normal((k, n)) + 1e-3 * rng.standard_normal((m, n))))
    U, S, VT = (torch.empty(c, dtype=torch.float64, device="cuda") for c in (m * k, k, k * n))
    rank, err = ctypes.c_int64(0), ctypes.c_double(0)
    for sh in ((100, 100), (6000, 40)):  # loads the kernels
        hb.svd(hb.to_device(np.asfortranarray(rng.standard_normal(sh))), *sh)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    free = torch.cuda.mem_get_info()[0]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    hb.check(hb.lib().heff_svd_d(p(A), m, n, k, 0.0, p(U), p(S), p(VT), ctypes.byref(rank), ctypes.byref(err), ctypes.c_void_p(st.cuda_stream)), "svd")
    st.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    assert rank.value == k
    assert used <= 1.25 * nbytes + (16 << 20), (used, nbytes)
