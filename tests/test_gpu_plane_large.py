"""Solves and the smoother of the FP64 plane kernels at their largest sizes (y and z in phases of their
own) against cuFFT's transforms: equal iteration counts, so they differ by rounding only (1e-12, as
at the smaller sizes)."""
import numpy as np
import pytest

from tests.gpu_common import FP64, gpu
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [208, 224, 240, 256])
def test_solve_and_smoother(n, monkeypatch):
    rng = np.random.default_rng(n)
    wm, u = rng.random(n ** 3), rng.random(n ** 3)
    out = []
    for path, kernel in (("", "k_plane"), ("0", "cufft_r2c_x3")):
        monkeypatch.setenv("GLIA_XPASS", path)
        g = gpu(n, FP64)
        g.set_tissue(wm)
        g.set_coefficients(k=0.05, rho=1.0)
        g.set_timing(True)
        c = u.copy()
        its = g.diffusion_solve(c, 0.01)
        assert g.timing()[kernel][0] > 0
        out.append((its, c, g.smooth(u, 0.3)))
        g.close()
    assert out[0][0] == out[1][0]
    assert rel_l2(out[0][1], out[1][1]) < 1e-12 and rel_l2(out[0][2], out[1][2]) < 1e-12


@pytest.mark.parametrize("n,plane", [(56, 0), (64, 1), (256, 1)])
def test_smoother_runs_on_the_plane_kernel_from_64(n, plane):
    g = gpu(n, FP64)
    g.set_timing(True)
    g.smooth(np.random.default_rng(n).random(n ** 3), 0.3)
    assert g.timing().get("k_plane", (0,))[0] == plane
    g.close()
