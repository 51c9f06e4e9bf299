"""The one-kernel Crank-Nicolson step with fewer, as many and more radial
levels than rows in flight, at both depths of the row ring, against the
separate kernels: the same expressions, so 1e-12 of each field's maximum."""
import numpy as np
import pytest

from calypso_b200 import PREC_FP64, configs
from test_gpu_cn import SLOTS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nr,nth,nph", [(7, 6, 12, 24), (7, 8, 12, 24), (15, 9, 24, 48), (31, 17, 48, 96),
                                          (127, 6, 128, 384), (127, 9, 128, 384)])
def test_ring_edges(L, nr, nth, nph):
    p = configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0, dt=1e-5)
    a, ea = run(p, PREC_FP64, 1, 3, 11)
    b, eb = run(p, PREC_FP64, 0, 3, 11)
    for q, s in enumerate(SLOTS):
        scale = max(np.max(np.abs(b[q])), 1e-300)
        assert np.max(np.abs(a[q] - b[q])) / scale <= 1e-12, s
    assert np.allclose(ea, eb, rtol=1e-12, atol=0.0)
