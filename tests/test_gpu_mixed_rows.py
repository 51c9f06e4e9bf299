"""The mixed-precision transforms around the edges of the operand kernels:
truncations on both sides of the 32- and 64-degree segments of the spectra
packing, radial counts that leave a partial block of levels, and Gauss grids
with one and several 16-byte groups of weights, against the oracle.

Tolerance 5e-6 relative L2, the repository's bar for the mixed transforms."""
import pytest

from calypso_b200 import PREC_MIXED, SphMHD, configs
from test_gpu_boundary import random_spec, rel_l2

pytestmark = pytest.mark.gpu

SHELLS = [(1, 5, 8, 8), (31, 6, 32, 72), (32, 7, 40, 96), (63, 5, 64, 144), (64, 6, 72, 162), (65, 5, 104, 192),
          (96, 9, 104, 216), (128, 5, 136, 288)]


@pytest.mark.parametrize("shell", SHELLS)
@pytest.mark.parametrize("nvec,nscal", [(4, 1), (1, 0), (0, 3)])
def test_transforms(oracle_lib, shell, nvec, nscal):
    L, nr, nth, nph = shell
    p = configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0)
    g, o = SphMHD(p, PREC_MIXED), oracle_lib.Oracle(p)
    nc = 3 * nvec + nscal
    spec = random_spec(L, nr, nc, 5, nvec)
    grid, grid_o = g.sph_back_trans(nvec, nscal, spec), o.sht_backward(nvec, nscal, spec)
    back, back_o = g.sph_forward_trans(nvec, nscal, grid_o), o.sht_forward(nvec, nscal, grid_o)
    for c in range(nc):
        assert rel_l2(grid[c], grid_o[c]) < 5e-6, c
        assert rel_l2(back[c], back_o[c]) < 5e-6, c
