"""The autotuner's FFT entry on grids with one FFT kernel to run: it has nothing to
choose and keeps its default; where there is a choice it is one of the kernels."""
import pytest

from calypso_b200 import PREC_FP64, PREC_MIXED, SphMHD, configs
from calypso_b200.sph_mhd import TUNE_FFT_THREADS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,shell,values", [
    (PREC_FP64, (21, 9, 40, 64), {384}),               # the general kernel alone
    (PREC_MIXED, (21, 9, 40, 64), {384}),
    (PREC_FP64, (21, 9, 48, 96), {384}),               # no four-step form at this truncation
    (PREC_MIXED, (21, 9, 48, 96), {512, 256, 128}),    # the Stockham kernel
    (PREC_FP64, (31, 9, 48, 96), {384, 512}),
    (PREC_MIXED, (31, 9, 48, 96), {384, 512, 256, 128}),
])
def test_fft_entry(prec, shell, values):
    g = SphMHD(configs.shell_params(*shell, E=1e-3, Ra=100.0), prec)
    for _ in range(3):
        assert g.autotune()[TUNE_FFT_THREADS] in values
    g.close()
