"""Float64 forward Legendre transform on grids with far more colatitudes than the
truncation needs: up to 21024 of them the kernel keeps the node weights in shared
memory, beyond that it reads them as it goes.

Compared with the sums over the library's own nodes, weights and functions
(cb2_gauss, cb2_plm) in numpy.  A sum of 2 nth terms, each of at most 16
roundings, differs by at most (2 nth + 16) 2^-53 of the terms' magnitudes on
either side."""
import numpy as np
import pytest

from calypso_b200 import PREC_FP64, SphMHD, configs, sph_tables
from calypso_b200.sph_mhd import rlm_size, rtm_size

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nth", [64, 21000, 21040])
def test_forward_sums(nth):
    L, nr, nph, nc = 8, 6, 18, 4                          # one vector, one scalar
    p = configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0)
    g = SphMHD(p, PREC_FP64)
    t = sph_tables(L, nr, nth, nph)
    assert rtm_size(t, nc) == (2 * L + 1) * nth * nr * nc and rlm_size(t, nc) == (L + 1) ** 2 * nr * nc
    f = np.random.default_rng(nth).standard_normal((2 * L + 1, nth, nr, nc))
    got = g.sel_forward_legendre_trans(nc, 1, 1, f.ravel(), t).reshape(nr, (L + 1) ** 2, nc)
    colat, w = g.gauss()
    r = p["r_icb"] + 0.5 * (p["r_cmb"] - p["r_icb"]) * (1.0 - np.cos(np.pi * np.arange(nr) / (nr - 1)))
    for l in range(L + 1):
        for m in range(-l, l + 1):
            P, dP = g.plm(l, abs(m))
            Pw, dPw, mPw = P * w, dP * w, abs(m) * P / np.sin(colat) * w
            sg = 1.0 if m >= 0 else -1.0
            g6 = (2 * l + 1) / (2.0 if m == 0 else 4.0)
            g7 = g6 / (l * (l + 1)) if l else 1.0
            R, T, F, S = (f[L + m, :, :, q] for q in range(4))
            To, Fo = f[L - m, :, :, 1], f[L - m, :, :, 2]
            terms = [(Pw[:, None] * R * g7 * r * r,),
                     (dPw[:, None] * T * g7 * r, -sg * mPw[:, None] * Fo * g7 * r),
                     (-sg * mPw[:, None] * To * g7 * r, -dPw[:, None] * F * g7 * r),
                     (Pw[:, None] * S * g6,)]
            for c, ts in enumerate(terms):
                ref = sum(x.sum(0) for x in ts)
                tol = 2 * (2 * nth + 16) * 2.0 ** -53 * sum(np.abs(x).sum(0) for x in ts)
                assert np.all(np.abs(got[:, l * l + l + m, c] - ref) <= tol), (l, m, c)
    g.close()
