"""The grid barriers of the FP64 solve kernels give up after a time limit. With a limit that runs out
at once every call that launches such a kernel reports it, none returns a field that was not
computed, and once the limit is restored the same context gives the results it gave before. Nothing
faults or hangs: the waiting CTAs record the fault and return."""
import numpy as np
import pytest

from glia_gb300 import _abi
from glia_gb300.context import GliaError
from tests.gpu_common import FP64, MIXED, configure, gpu, small_problem
from tests.helpers import reference_test_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 160])  # planes in shared memory, y and z phases of their own
def test_a_wait_that_runs_out_is_reported_by_every_call(n):
    wl, tissue, centers = small_problem(n, 2, n_gauss=4)
    g = gpu(n, FP64)
    # the reference's rule takes the preconditioner's dt from the solve before, another one after
    # other calls; the dt is taken when the coefficients are set
    g.set_pcg(pc_dt_mode=_abi.GLIA_PC_DT_FIXED, pc_dt=0.005)
    configure(g, wl, tissue, centers)
    x = np.concatenate([np.linspace(0.1, 0.9, len(centers)), [wl.kappa, wl.rho]])
    d1 = (reference_test_field(n) > 0.3).astype(np.float64)
    direction = np.linspace(-1.0, 1.0, x.size)

    def solve():
        c = reference_test_field(n)
        g.diffusion_solve(c, 0.01)
        return c

    def evaluate():
        J, dJ = g.eval_objective_and_gradient(x, d1)
        return np.concatenate([[J], dJ])

    calls = [lambda: g.apply_d(reference_test_field(n)), solve,
             lambda: g.smooth(reference_test_field(n), 0.3),
             lambda: g.solve_state(reference_test_field(n)), evaluate,
             lambda: g.hessian_matvec(direction)]
    before = [np.array(call()) for call in calls]
    for call in calls:
        if call is calls[-1]:  # needs a state history
            evaluate()
        assert g.api.selftest_wait_limit(g._h, -1) == _abi.GLIA_OK
        for _ in range(2):
            with pytest.raises(GliaError, match="GLIA_ERR_CUDA"):
                call()
        assert g.api.selftest_wait_limit(g._h, 0) == _abi.GLIA_OK
    for call, want in zip(calls, before):
        assert np.array_equal(call(), want)
    g.close()


def test_contexts_without_such_a_kernel_refuse():
    g = gpu(32, MIXED)
    assert g.api.selftest_wait_limit(g._h, -1) == _abi.GLIA_ERR_INVALID
    g.close()
