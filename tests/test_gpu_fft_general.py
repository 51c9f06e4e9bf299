"""The products kernels of the zonal transform in single precision over grids
of every radix pair, and the float64 kernels of 768 points over truncations
(L = 255 takes the four-step one), against numpy.

Tolerances, relative L2 per product.  float64: 1e-12, the repository's bar for
float64 transforms.  Single precision: a forward and a backward transform of
at most 20 dependent roundings a point each (2^-24 apiece, random signs: below
5e-7 together), the rounding of input and output, and for the products the
cancellation of a difference of two products (a factor of up to 2): 2e-6."""
import pytest

from calypso_b200 import PREC_FP64, PREC_MIXED, SphMHD, configs
from test_gpu_boundary import (BALANCED, SKEWED, _products, four_to_rtm, np_fft_backward, np_fft_forward, random_four,
                               rel_l2, rtm_to_four, tables_for)

pytestmark = pytest.mark.gpu


def check(prec, L, nr, nth, nph, scales, tol):
    p = configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0)
    g = SphMHD(p, prec)
    t = tables_for(p, 8)
    four = random_four(L, nr, nth, 13, 17, scales=scales)
    got = rtm_to_four(g.fft_products(four_to_rtm(four, t, 13), t), t, 12, 12, L)
    prod = _products(np_fft_backward(four, nph), p["coef_velo"], p["coef_lor"], p["coef_induct"], p["coef_temp"])
    want = np_fft_forward(prod, L)
    for c in range(12):
        assert rel_l2(got[c], want[c]) < tol, (c, rel_l2(got[c], want[c]))


@pytest.mark.parametrize("L,nth,nph", [(1, 8, 4), (2, 8, 6), (5, 8, 12), (7, 16, 16), (15, 24, 48), (21, 32, 64),
                                       (20, 24, 54), (20, 24, 72), (35, 56, 108), (42, 64, 128), (40, 48, 162),
                                       (85, 128, 256), (100, 152, 324), (20, 24, 972), (20, 24, 1024)])
def test_single(L, nth, nph):
    check(PREC_MIXED, L, 5, nth, nph, BALANCED, 2e-6)


@pytest.mark.parametrize("L,nr,nth", [(1, 5, 4), (20, 7, 24), (127, 5, 128), (254, 5, 256), (255, 6, 256)])
def test_double_768(L, nr, nth):
    check(PREC_FP64, L, nr, nth, 768, SKEWED, 1e-12)
