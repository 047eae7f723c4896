"""The counters of a context (glia_stats) are those of the calls made, whichever kernels served them:
FP64 contexts with plane kernels and with cuFFT's transforms count the same."""
import numpy as np
import pytest

from tests.gpu_common import FP64, configure, gpu, small_problem
from tests.helpers import reference_test_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("history", [(0, 0), (1, 2)])  # full, checkpointed
def test_counters_do_not_depend_on_the_path(history, monkeypatch):
    n = 32
    wl, tissue, centers = small_problem(n, 3, n_gauss=4)
    x = np.concatenate([np.linspace(0.1, 0.9, len(centers)), [wl.kappa, wl.rho]])
    f = reference_test_field(n)
    out = []
    for path in ("", "0"):
        monkeypatch.setenv("GLIA_XPASS", path)
        g = gpu(n, FP64)
        configure(g, wl, tissue, centers, *history)
        # cuFFT's path also counts the six transforms of the loop that its first solve records
        g.diffusion_solve(f.copy(), 0.01)
        g.reset_stats()
        seen = []
        for call in (lambda: g.apply_d(f), lambda: g.smooth(f, 0.3),
                     lambda: g.diffusion_solve(f.copy(), 0.01), lambda: g.solve_state(f),
                     lambda: g.eval_objective_and_gradient(x, (f > 0.3).astype(np.float64)),
                     lambda: g.hessian_matvec(x)):
            call()
            # of the last solve: a real number, and one that the kappa gradient's D apply clears
            # on cuFFT's path
            seen.append({k: v for k, v in g.stats().items()
                         if k not in ("last_rnorm", "last_ksp_itr")})
        out.append(seen)
        g.close()
    assert out[0] == out[1]
