"""The maximised likelihood does not depend on the template's scale: two lags that are nearly equal, told apart
by the FP64 values, for templates so faint that |g|^2 is below FP32's range."""
import numpy as np
import pytest

import gw_analysis_tools_gb300 as G
from gw_analysis_tools_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [15680, 16411])  # a direct transform, a padded one
@pytest.mark.parametrize("scale", [1.0, 1e20, 1e23, 1e24, 1e25, 1e26])
def test_faint_templates(gpu_ctx, oracle, N, scale):
    T = 16
    f = 20.0 + np.arange(N) / T
    psd = W.analytic_psd(f)
    src = W.config1_source()
    # the draw's own waveform, arriving half a sample off the lags: the two next to it differ by 4e-8 .. 1e-6
    hp, _ = oracle.fourier_waveform(f, oracle.params_from_dict(dict(src, RA=0.0, DEC=0.0, psi=0.0, phiRef=1.0, incl_angle=0.0,
                                                                    tc=1.0, f_ref=10.0)), oracle.IMRPhenomD)
    faint = dict(src, Luminosity_Distance=src["Luminosity_Distance"] * scale)
    for off in (1e-7, -1e-7, 3e-7, -3e-7, 1e-6, -1e-6, 3e-6, -3e-6):
        data = hp * np.exp(2j * np.pi * np.arange(N) * (100.5 + off) / N)
        h = gpu_ctx.register_data("Hanford", f, data, psd)
        ref = oracle.maximized_loglik_intrinsic(faint, f, [data], [psd], approximant=0)
        out, st = gpu_ctx.maximized_loglik_batch(G.params_array([faint]), [h], 0)
        gpu_ctx.release_data(h)
        assert st[0] == 0 and abs(out[0] - ref) <= 1e-9 * abs(ref), (off, out[0] / ref - 1)
