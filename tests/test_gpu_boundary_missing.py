"""A table of full length that lists one mode twice leaves another out, and that
one is zero in the backward transform, whatever an earlier call left in the work
fields: the result is that of the shorter table without the missing mode."""
import numpy as np
import pytest

from calypso_b200 import PREC_FP64, PREC_MIXED, SphMHD, configs, sph_tables
from calypso_b200.sph_mhd import rlm_size
from test_gpu_boundary import random_spec, spec_to_rlm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("gone", [(0, 0), (3, -2), (7, 7)])
def test_mode_listed_twice(prec, gone):
    L, nr, nth, nph = 7, 5, 16, 24
    g = SphMHD(configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0), prec)
    modes = [(l, m) for l in range(L + 1) for m in range(-l, l + 1)]
    short = [x for x in modes if x != gone]
    twice = short + [short[5]]
    spec = random_spec(L, nr, 4, 3, 1)
    out = []
    for jo in (short, twice):
        full = sph_tables(L, nr, nth, nph)
        WR = spec_to_rlm(10.0 * spec, full, 4)
        assert WR.size == rlm_size(full, 4)
        g.sel_backward_legendre_trans(4, 1, 1, WR, full)          # fills every work field
        t = sph_tables(L, nr, nth, nph, j_order=jo)
        out.append(g.sel_backward_legendre_trans(4, 1, 1, spec_to_rlm(spec, t, 4), t))
    assert np.array_equal(*out)
