"""Complex tensors that are not 16-byte aligned are refused before anything is launched, at the sizes of the one-launch product and at
those of the four kernels (the addresses are never read)."""
import ctypes

import pytest

import dmrg_b200 as hb


@pytest.mark.parametrize("chi", [16, 300])
@pytest.mark.parametrize("which", ["mps", "mpo", "envL", "envR"])
def test_misaligned_complex_tensors(chi, which):
    L = hb.lib()
    p = {n: ctypes.c_void_p(0x10000 * (i + 1) + (8 if n == which else 0)) for i, n in enumerate(["mps", "mpo", "envL", "envR"])}
    ten = (p["mps"], hb.dims((4, chi, chi)), p["mpo"], hb.dims((3, 3, 4, 4)), p["envL"], hb.dims((chi, chi, 3)), p["envR"], hb.dims((chi, chi, 3)))
    out = (ctypes.c_double * 2)()
    assert L.heff_matvec_z(ctypes.c_void_p(0x100000), *ten, None) == 7  # HEFF_BAD_ARG
    assert L.heff_expval_z(out, *ten, None) == 7  # HEFF_BAD_ARG
