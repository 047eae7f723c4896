"""FP64 contexts in a captured batch: the preconditioner of a graph's solves is that of its own
parameters, whatever was captured, launched or solved on the context before, and an ordinary solve
after a launch uses its own. Results equal a fresh context's bit for bit: a solve that stops on
another preconditioner differs by the PCG tolerance (1e-6), far above rounding."""
from types import SimpleNamespace

import numpy as np
import pytest

from glia_gb300 import _abi
from glia_gb300.batch import GraphBatch
from tests.gpu_common import FP64, configure, gpu, small_problem
from tests.helpers import reference_test_field

pytestmark = pytest.mark.gpu
SIZES, NT, KAPPAS = (24, 32), 2, (0.02, 0.3)


def inputs(n):
    wl, tissue, centers = small_problem(n, NT, n_gauss=4)
    d1 = (reference_test_field(n) > 0.3).astype(np.float64)
    xs = [np.concatenate([np.linspace(0.1, 0.9, len(centers)), [k, wl.rho]]) for k in KAPPAS]
    return wl, tissue, centers, d1, xs


def context(n):
    wl, tissue, centers, _, _ = inputs(n)
    ctx = gpu(n, FP64)
    configure(ctx, wl, tissue, centers)
    ctx.set_pcg(pc_dt_mode=_abi.GLIA_PC_DT_MATCHED)
    return ctx


def fresh(n, x, d1):
    ctx = context(n)
    out = ctx.eval_objective_and_gradient(x, d1)
    ctx.close()
    return out


def fresh_solve(n, x, d1, dt):
    ctx = context(n)
    ctx.eval_objective_and_gradient(x, d1)
    c = reference_test_field(n)
    its = ctx.diffusion_solve(c, dt)
    ctx.close()
    return its, c


@pytest.fixture
def batch():
    """A graph captured, but never launched, at the first kappa."""
    data = [inputs(n) for n in SIZES]
    b = SimpleNamespace(ctxs=[context(n) for n in SIZES],
                        problems=[SimpleNamespace(n=n, x=d[4][0]) for n, d in zip(SIZES, data)],
                        data=[d[3] for d in data])
    g = GraphBatch(b)
    for p, d in zip(b.problems, data):
        p.x = d[4][1]
    yield g
    g.close()
    for c in b.ctxs:
        c.close()


def check(g):
    for p, d1, (J, dJ) in zip(g.batch.problems, g.batch.data, g.evaluate()[1]):
        want = fresh(p.n, p.x, d1)
        assert J == want[0] and np.array_equal(dJ, want[1])


def test_captured_twice_before_the_first_launch(batch):
    batch.capture()
    batch.capture()
    check(batch)
    check(batch)


def test_solves_between_capture_and_launch_and_after(batch):
    batch.capture()
    for _ in range(2):
        for p, c in zip(batch.batch.problems, batch.batch.ctxs):
            c.diffusion_solve(reference_test_field(p.n), 0.1)
        check(batch)
        for p, c, d1 in zip(batch.batch.problems, batch.batch.ctxs, batch.batch.data):
            u = reference_test_field(p.n)
            its = c.diffusion_solve(u, 0.1)
            want = fresh_solve(p.n, p.x, d1, 0.1)
            assert its == want[0] and np.array_equal(u, want[1])
