"""The plane kernels (plane.cuh) at every grid size they cover, in both precisions: D apply and the
smoother against numpy's FFT in double, one diffusion solve and a two-step state / gradient
against the separate transform paths of the same library (GLIA_XPASS=0: cuFFT).

Tolerances. D apply in double: numpy's own FFT errors, 2 transforms of log2 n^3 stages at 1.1e-16
each, amplified by two derivatives of up to n/2 on fields whose spectrum is flat: 1e-13 relative
to the result's norm. In float the same at 6e-8: 5e-6. The solves stop at 1e-6 of the right-hand
side, with equal iteration counts, so the two paths differ by rounding only: 1e-12 and 1e-5."""
import numpy as np
import pytest

from glia_gb300 import synthetic as syn
from tests.gpu_common import FP64, MIXED, configure, gpu, small_problem
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu
SIZES = {FP64: [*range(16, 129, 8), 144, 160, 176, 192, 208, 224, 240, 256],
         MIXED: [*range(16, 129, 8), 144, 160, 176, 192, 208, 224]}
CASES = [(p, n) for p in (FP64, MIXED) for n in SIZES[p]]


def field(n, seed=0):
    return np.random.default_rng(seed).random(n ** 3)


def numpy_d(u, k, n):
    w = np.fft.fftfreq(n, 1 / n)
    w[n // 2] = 0
    ws = (w[:, None, None], w[None, :, None], w[None, None, : n // 2 + 1])
    s = np.fft.rfftn(u.reshape((n,) * 3))
    out = 0
    for wj in ws:
        g = np.fft.irfftn(1j * wj * s, s=(n,) * 3, axes=(0, 1, 2)) * k
        out = out + np.fft.irfftn(1j * wj * np.fft.rfftn(g), s=(n,) * 3, axes=(0, 1, 2))
    return out.reshape(-1)


@pytest.mark.parametrize("prec,n", CASES)
def test_d_apply_against_numpy(prec, n):
    rng = np.random.default_rng(n)
    wm = rng.random((n, n, n))
    g = gpu(n, prec)
    g.set_tissue(wm.reshape(-1))
    g.set_coefficients(k=0.05, rho=1.0)
    u = field(n)
    if prec == MIXED:  # what the float context holds
        u, wm = u.astype(np.float32).astype(np.float64), wm.astype(np.float32).astype(np.float64)
    got = g.apply_d(u)
    assert rel_l2(got, numpy_d(u, 0.05 * wm, n)) < (1e-13 if prec == FP64 else 5e-6)
    g.close()


@pytest.mark.parametrize("prec,n", [c for c in CASES if c[1] <= 192])
def test_solve_state_and_gradient_match_the_cufft_path(prec, n, monkeypatch):
    if n < 32:  # too coarse for the seeded white matter: the whole brain mask instead
        wl = syn.GradientWorkload(n=n, nt=2, n_gauss=4)
        m = syn.ellipsoid_mask(n)
        tissue = syn.Tissue(wm=m * 1.0, gm=m * 0.0, csf=m * 0.0, vt=m * 0.0, mask=m)
        centers = np.pi + 0.4 * np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, -1.0]])
    else:
        wl, tissue, centers = small_problem(n, 2, n_gauss=4)
    x = np.concatenate([np.linspace(0.1, 0.9, 4), [wl.kappa, wl.rho]])
    d1 = (field(n, 1) > 0.5).astype(np.float64)
    out = []
    for path in ("", "0"):
        monkeypatch.setenv("GLIA_XPASS", path)
        g = gpu(n, prec)
        configure(g, wl, tissue, centers)
        c = field(n, 2)
        its = g.diffusion_solve(c, 0.01)
        s = g.smooth(field(n, 3), 0.3)
        J, dJ = g.eval_objective_and_gradient(x, d1)
        out.append((its, c, s, g.solve_state(field(n, 4) * 0.9), np.array([J]), dJ))
        g.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert rel_l2(a, b) < (1e-12 if prec == FP64 else 1e-5)


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_non_finite_fields_are_reported(prec):
    """A NaN or an infinity in the field stops the solve with an error, as on the other paths."""
    from glia_gb300.context import GliaError

    for bad in (np.nan, np.inf):
        g = gpu(32, prec)
        g.set_tissue(np.ones(32 ** 3))
        g.set_coefficients(k=0.05, rho=1.0)
        c = field(32)
        c[1234] = bad
        with pytest.raises(GliaError, match="NOT_CONVERGED"):
            g.diffusion_solve(c, 0.01)
        c = field(32)
        g.diffusion_solve(c, 0.01)  # the context stays usable
        assert np.isfinite(c).all()
        g.close()
