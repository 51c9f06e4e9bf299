"""The routine-level entry points give the same values whatever the strides
and the order of the caller's tables: the layouts with the radius running
fastest and those with the order fastest go through different kernels, and
only move values, so the results are compared for equality."""
import numpy as np
import pytest

from calypso_b200 import PREC_FP64, PREC_MIXED, SphMHD, configs, sph_tables
from calypso_b200.sph_mhd import rlm_size, rtm_size
from test_gpu_boundary import four_to_rtm, random_four, random_spec, rlm_to_spec, rtm_to_four, spec_to_rlm

pytestmark = pytest.mark.gpu

# (L, nr, nth, nph): one radial tile and a remainder, odd truncations
SHELLS = [(7, 5, 16, 24), (21, 9, 40, 64), (31, 33, 48, 96)]


def tables(shell, seed, order, drop):
    """k_fast: the default strides and mode order; m_fast: the orders fastest
    in rtm, k fastest in rlm, both orders shuffled.  drop: leave out every
    seventh mode and fifth order."""
    L, nr, nth, nph = shell
    jo = [(l, m) for l in range(L + 1) for m in range(-l, l + 1)]
    mo = list(range(-L, L + 1))
    if drop:
        jo = [x for i, x in enumerate(jo) if i % 7 != 3]
        mo = [m for i, m in enumerate(mo) if i % 5 != 2]
    if order == "k_fast":
        return sph_tables(L, nr, nth, nph, j_order=jo, m_order=mo)
    rng = np.random.default_rng(seed)
    jo = [jo[i] for i in rng.permutation(len(jo))]
    mo = [mo[i] for i in rng.permutation(len(mo))]
    nm = len(mo)
    return sph_tables(L, nr, nth, nph, j_order=jo, m_order=mo, istep_rlm=(1, nr), istep_rtm=(nm, nm * nr, 1))


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("shell", SHELLS)
@pytest.mark.parametrize("nvec,nscal,extra,drop", [(3, 2, 0, False), (1, 0, 2, True), (0, 3, 0, False), (5, 1, 1, True)])
def test_layouts_agree(prec, shell, nvec, nscal, extra, drop):
    L, nr, nth, nph = shell
    g = SphMHD(configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0), prec)
    nc = 3 * nvec + nscal
    ncomp, tail = nc + extra, 5
    spec = random_spec(L, nr, nc, 3, nvec)
    four = random_four(L, nr, nth, nc, 4)
    got = []
    for order in ("k_fast", "m_fast"):
        t = tables(shell, 11, order, drop)
        n_rtm, n_rlm = rtm_size(t, ncomp), rlm_size(t, ncomp)
        # the call clears its output, beyond the tables' extent too
        WS = np.full(n_rtm + tail, 7.0)
        g.sel_backward_legendre_trans(ncomp, nvec, nscal, spec_to_rlm(spec, t, ncomp), t, WS=WS)
        assert not WS[n_rtm:].any()
        if extra:
            assert not WS[:n_rtm].reshape(-1, ncomp)[:, nc:].any()
        WS2 = np.full(n_rlm + tail, 7.0)
        g.sel_forward_legendre_trans(ncomp, nvec, nscal, four_to_rtm(four, t, ncomp), t, WS=WS2)
        assert not WS2[n_rlm:].any()
        F = g.back_MHD_FFT_sel_from_recv(nc, four_to_rtm(four, t, nc), t)
        WS3 = g.fwd_MHD_FFT_sel_from_recv(nc, F, t)
        got.append([rtm_to_four(WS, t, ncomp, nc, L), rlm_to_spec(WS2, t, ncomp, nc, g.jmax), F,
                    rtm_to_four(WS3, t, nc, nc, L)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_products_layouts_agree(prec):
    shell = (21, 9, 40, 64)
    L, nr, nth, nph = shell
    g = SphMHD(configs.shell_params(L, nr, nth, nph, E=1e-3, Ra=100.0), prec)
    four = random_four(L, nr, nth, 13, 4)
    a, b = (rtm_to_four(g.fft_products(four_to_rtm(four, t, 13), t), t, 12, 12, L)
            for t in (tables(shell, 11, o, False) for o in ("k_fast", "m_fast")))
    assert np.array_equal(a, b)
