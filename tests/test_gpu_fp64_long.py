"""Long FP64 simulations keep cuFFT's transforms: rounding in tumour-free tissue grows like
exp(rho T), so beyond rho T = 10.5 the plane kernels' answers would leave cuFFT's by more than FP64
results may move (1e-9 of their norm). Below, both paths agree to that bound; above, they are one
path and agree bit for bit."""
import numpy as np
import pytest

from tests.gpu_common import FP64, configure, gpu, small_problem
from tests.helpers import reference_test_field, rel_l2

pytestmark = pytest.mark.gpu
N, NT, KAPPA = 32, 100, 0.01


def run(rho):
    wl, tissue, centers = small_problem(N, NT, n_gauss=8)
    g = gpu(N, FP64)
    configure(g, wl, tissue, centers)
    x = np.concatenate([np.linspace(0.0, 0.9, len(centers)), [KAPPA, rho]])
    g.set_timing(True)
    J, dJ = g.eval_objective_and_gradient(x, (reference_test_field(N) > 0.3).astype(np.float64))
    plane = g.timing().get("k_plane", (0,))[0]
    c1 = g.get_state(NT)
    g.close()
    return c1, np.concatenate([[J], dJ]), plane, rho * tissue.wm.max() * NT * wl.dt


@pytest.mark.parametrize("rho,long", [(9.0, False), (14.0, True)])
def test_results_stay_with_cufft(rho, long, monkeypatch):
    c1, gradient, plane, growth = run(rho)
    assert (growth > 10.5) == long and (plane == 0) == long
    monkeypatch.setenv("GLIA_XPASS", "0")
    c1_cufft, gradient_cufft, plane, _ = run(rho)
    assert plane == 0
    for a, b in ((c1, c1_cufft), (gradient, gradient_cufft)):
        if long:
            assert np.array_equal(a, b)
        else:
            assert rel_l2(a, b) <= 1e-9
