"""The float64 transforms at the edges of their tiles against the oracle and
numpy: odd hemispheres (8-byte table copies), one partial node tile and one
node beyond a full one, degrees around the 32- and 64-degree row tiles, column
remainders, and every radix of the products kernel with the smallest and the
largest zonal grids (with and without row padding).

Tolerance 1e-12 relative L2, the repository's bar for float64 transforms (the
same sums in another order: at most a few hundred terms of 1.1e-16)."""
import numpy as np
import pytest

from calypso_b200 import PREC_FP64, SphMHD, configs
from test_gpu_boundary import (SKEWED, _products, four_to_rtm, np_fft_backward, np_fft_forward, random_four,
                               random_spec, rel_l2, rtm_to_four, tables_for)

pytestmark = pytest.mark.gpu

SHELLS = [(1, 5, 4, 4), (5, 6, 8, 12), (15, 7, 24, 48), (21, 5, 34, 64), (31, 9, 48, 96), (32, 5, 66, 108),
          (63, 5, 98, 192), (64, 6, 100, 216), (106, 5, 162, 324)]


@pytest.mark.parametrize("shell", SHELLS)
@pytest.mark.parametrize("nvec,nscal", [(4, 1), (1, 0), (0, 3)])
def test_transforms(oracle_lib, shell, nvec, nscal):
    L, nr, nth, nph = shell
    p = configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0)
    g, o = SphMHD(p, PREC_FP64), oracle_lib.Oracle(p)
    nc = 3 * nvec + nscal
    spec = random_spec(L, nr, nc, 5, nvec)
    grid, grid_o = g.sph_back_trans(nvec, nscal, spec), o.sht_backward(nvec, nscal, spec)
    back, back_o = g.sph_forward_trans(nvec, nscal, grid_o), o.sht_forward(nvec, nscal, grid_o)
    for c in range(nc):
        assert rel_l2(grid[c], grid_o[c]) < 1e-12, c
        assert rel_l2(back[c], back_o[c]) < 1e-12, c


@pytest.mark.parametrize("L,nth,nph", [(1, 4, 4), (2, 4, 6), (5, 8, 12), (15, 24, 48), (21, 32, 64), (20, 24, 72),
                                       (35, 54, 108), (42, 64, 128), (40, 48, 162), (20, 24, 256), (20, 24, 324),
                                       (20, 24, 972), (20, 24, 1024)])
def test_products(L, nth, nph):
    p = configs.shell_params(L, 5, nth, nph, E=1e-3, Ra=100.0)
    g = SphMHD(p, PREC_FP64)
    t = tables_for(p, 8)
    four = random_four(L, 5, nth, 13, 31, scales=SKEWED)
    got = rtm_to_four(g.fft_products(four_to_rtm(four, t, 13), t), t, 12, 12, L)
    prod = _products(np_fft_backward(four, nph), p["coef_velo"], p["coef_lor"], p["coef_induct"], p["coef_temp"])
    want = np_fft_forward(prod, L)
    for c in range(12):
        assert rel_l2(got[c], want[c]) < 1e-12, (c, rel_l2(got[c], want[c]))
