"""The Gaussian of every two-band colour term, 2^(-t^2 / 64), by itself: within
1.5e-15 of the CUDA library exp2 (two units in the last place each for the
table's and the reference's exp2, half a unit for the polynomial's last two
steps, the product and the reference's own), over both signs, the table's
boundaries and the whole range; nothing beyond the cap."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi,tol", [
    (0.0, 1.0, 1.5e-15), (-8.0, 8.0, 1.5e-15), (8.0, 64.0, 1.5e-15), (-255.5, -60.0, 1.5e-15),
    (60.0, 255.5, 1.5e-15), (255.0, 255.7, 1.5e-15), (256.0, 300.0, 0.0), (-1e300, -256.0, 0.0)])
def test_gauss_table(gpu_ctx, lo, hi, tol):
    from pofd_affine_b200._lib import support_lib
    out = C.c_double()
    assert support_lib().pofd_exp2_gauss_check(0, 1 << 21, lo, hi, C.byref(out)) == 0
    assert out.value <= tol
