"""The FP64 plane kernels (64-bit fixed point between the transforms) against long double: a D apply
and a simulation are no further from the exact result than the same with cuFFT's FP64 transforms
(GLIA_XPASS=0). The reference applies derivatives and preconditioner as matrices along each axis, in
long double (64 bits of mantissa or more), and stops PCG where the library does."""
import numpy as np
import pytest

from tests.gpu_common import FP64, gpu
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu
LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")


def along(m, f, axis):
    return np.moveaxis(np.tensordot(m, f, axes=(1, axis)), 0, axis)


class Exact:
    def __init__(self, n, k):
        i = np.arange(n)
        j = (i[:, None] - i[None, :]) % n
        waves = np.arange(1, n // 2)
        angle = 2 * PI * ((waves[:, None, None] * j) % n).astype(LD) / n
        self.d = -2 * (waves[:, None, None].astype(LD) * np.sin(angle)).sum(0) / n
        # orthonormal real Fourier basis, one row per function, and its squared wave numbers
        a = 2 * PI * ((waves[:, None] * i) % n).astype(LD) / n
        one = np.ones((1, n), LD)
        self.q = np.concatenate([one, np.sqrt(LD(2)) * np.cos(a), np.sqrt(LD(2)) * np.sin(a),
                                 one * (1 - 2 * (i % 2))]) / np.sqrt(LD(n))
        w2 = np.concatenate([[0], waves, waves, [0]]).astype(LD) ** 2
        self.w2 = w2[:, None, None] + w2[None, :, None] + w2[None, None, :]
        self.k = k.astype(LD)

    def apply_d(self, u):
        return sum(along(self.d, self.k * along(self.d, u, x), x) for x in range(3))

    def precondition(self, u, c):
        for x in range(3):
            u = along(self.q, u, x)
        u = u / (1 + c * self.w2)
        for x in range(3):
            u = along(self.q.T, u, x)
        return u

    def solve(self, c, dt, pc):
        a = LD(0.5) * dt
        d = self.apply_d(c)
        x, r, b = c.copy(), 2 * a * d, c + a * d
        stop = LD(1e-6) * np.sqrt((self.precondition(b, pc) ** 2).sum())
        z = self.precondition(r, pc)
        p, beta = z, (z * r).sum()
        for _ in range(50):
            w = p - a * self.apply_d(p)
            alpha = beta / (p * w).sum()
            x, r = x + alpha * p, r - alpha * w
            z = self.precondition(r, pc)
            if np.sqrt((z * z).sum()) <= stop:
                return x
            beta, old = (z * r).sum(), beta
            p = z + beta / old * p
        raise AssertionError("not converged")


def smooth_field(n, seed):
    i = 2 * np.pi * np.arange(n) / n
    rng = np.random.default_rng(seed)
    f = np.ones((n, n, n))
    for x in range(3):
        g = sum(rng.uniform(-0.4, 0.4) * np.cos(m * i + rng.uniform(0, 6)) for m in (1, 2, 3))
        f = f * (1 + g / 2).reshape([-1 if x == y else 1 for y in range(3)])
    return f / f.max()


def errors(call, want, monkeypatch):
    out = []
    for path in ("", "0"):
        monkeypatch.setenv("GLIA_XPASS", path)
        got = call().astype(LD) - want.reshape(-1)
        out.append(float(np.sqrt((got ** 2).sum() / (want ** 2).sum())))
    print("off long double: plane kernel %.2e, cuFFT %.2e" % tuple(out))
    return out


@pytest.mark.parametrize("field,exponent", [("smooth", 0), ("white", 0), ("white", -900),
                                            ("white", 900)])
@pytest.mark.parametrize("n", [16, 24, 32])
def test_d_apply(n, field, exponent, monkeypatch):
    """Also of fields near the ends of double's range: blocks carry their exponents."""
    wm = smooth_field(n, 1)
    u = smooth_field(n, 2) if field == "smooth" else np.random.default_rng(n).standard_normal(
        (n, n, n))
    u = np.ldexp(u, exponent)
    k = 0.0625  # a power of two: the diffusivity field is exact

    def call():
        g = gpu(n, FP64)
        g.set_tissue(wm.reshape(-1))
        g.set_coefficients(k=k, rho=1.0)
        out = g.apply_d(u.reshape(-1))
        g.close()
        return out

    here, cufft = errors(call, Exact(n, k * wm).apply_d(u.astype(LD)), monkeypatch)
    assert here <= cufft


@pytest.mark.parametrize("n", [16, 24])
def test_simulation(n, monkeypatch):
    """Six Strang steps with a fixed preconditioner."""
    nt, dt, k, rho, pc_dt = 6, 0.015625, 0.0625, 8.0, 0.0078125
    wm = smooth_field(n, 3)
    c0 = smooth_field(n, 4) ** 4 / 2

    def call():
        g = gpu(n, FP64)
        g.set_time(dt, nt)
        g.set_pcg(pc_dt_mode=1, pc_dt=pc_dt)
        g.set_tissue(wm.reshape(-1))
        g.set_coefficients(k=k, rho=rho)
        out = g.solve_state(c0.reshape(-1))
        g.close()
        return out

    e = Exact(n, k * wm)
    pc = LD(0.25) * LD(pc_dt) * LD((k * wm).sum() / (wm > 0.1).sum())
    growth = np.exp(LD(rho) * wm.astype(LD) * LD(dt))
    c = c0.astype(LD)
    for _ in range(nt):
        c = e.solve(c, LD(dt) / 2, pc)
        c = c * growth / (c * growth + 1 - c)
        c = e.solve(c, LD(dt) / 2, pc)
    here, cufft = errors(call, c, monkeypatch)
    assert cufft < 1e-12  # the reference follows the same iteration
    assert here <= cufft


def test_reference_is_the_spectral_derivative():
    n = 16
    e = Exact(n, np.ones((n, n, n)))
    u = np.random.default_rng(0).standard_normal((n, n, n))
    w = np.fft.fftfreq(n, 1 / n)
    w[n // 2] = 0
    want = np.fft.ifft(1j * w[:, None, None] * np.fft.fft(u, axis=0), axis=0).real
    assert rel_l2(along(e.d, u.astype(LD), 0).astype(float), want) < 1e-13
